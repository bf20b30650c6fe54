"""The U-Net kernels at the edges of their tiles: weight and bias gradients
over partial pixel tiles and every channel-tile shape, the mma.sync
convolution on every tile it picks, the vector and scalar forms of the
pooling and upsampling maps."""
import pytest

torch = pytest.importorskip("torch")
import torch.nn.functional as F  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _rand(*shape, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(*shape, device="cuda", generator=g).bfloat16()


def _torch_w(w, co, ci):
    return w.view(3, 3, co, ci).permute(2, 3, 0, 1)


# widths below, at and above a 16- and a 32-column tile; rows that end inside a tile; 16 x 16, 16 x 32, 32 x 16 and
# 32 x 32 channel tiles with the two inputs split inside one; several tiles per block; one pixel
@pytest.mark.parametrize("n,h,w,c0,c1,co", [
    (1, 1, 1, 16, 0, 16), (2, 17, 9, 16, 0, 48), (1, 16, 16, 32, 0, 16), (2, 9, 17, 16, 16, 32), (1, 7, 33, 16, 32, 32),
    (3, 33, 31, 64, 32, 64), (2, 8, 64, 128, 0, 128), (8, 257, 70, 16, 0, 16)])
def test_weight_and_bias_gradient_tiles(n, h, w, c0, c1, co):
    """Against torch in 64 bits on the same bf16 values.  The products are
    exact in FP32; an FP32 sum of N of them in any order is off by at most
    N 2^-24 of the sum of their sizes, and for random signs by far less than
    the 1e-5 of the result's norm asked here."""
    from seispie_b200 import _lib
    from seispie_b200.engine import check, ptr, stream_handle
    lib, st = _lib.load(), stream_handle(None)
    x0, x1, g = _rand(n, h, w, c0, seed=1), _rand(n, h, w, max(c1, 16), seed=2), _rand(n, h, w, co, seed=3)
    ct = c0 + c1
    part = torch.full((lib.fwi_unet_wgrad_partials(co, ct, n, h, w),), float("nan"), device="cuda")
    dw, db = torch.empty(9 * co * ct, device="cuda"), torch.empty(co, device="cuda")
    check(lib.fwi_unet_conv3x3_wgrad(ptr(g), co, ptr(x0), c0, ptr(x1) if c1 else None, c1, n, h, w, ptr(part), ptr(dw),
                                     ptr(db), st), "wgrad")
    x = torch.cat([x0, x1[..., :c1]], -1).double().permute(0, 3, 1, 2)
    wt = torch.zeros(co, ct, 3, 3, dtype=torch.float64, device="cuda", requires_grad=True)
    F.conv2d(x, wt, padding=1).backward(g.double().permute(0, 3, 1, 2))
    got = _torch_w(dw, co, ct).double()
    assert float((got - wt.grad).norm()) <= 1e-5 * float(wt.grad.norm())
    ref = g.double().sum((0, 1, 2))
    assert float((db.double() - ref).norm()) <= 1e-5 * float(g.double().abs().sum((0, 1, 2)).norm())


# 128 x 64, 64 x 64, 64 x 32, 128 x 32, 128 x 16 and 64 x 16 tiles of pixels x channels
@pytest.mark.parametrize("n,h,w,c0,c1,co", [
    (8, 80, 62, 16, 0, 64), (4, 61, 63, 32, 16, 128), (8, 32, 16, 128, 0, 128), (8, 80, 62, 16, 0, 32),
    (9, 80, 62, 16, 16, 16), (1, 5, 3, 16, 0, 48)])
def test_narrow_convolution_tiles(n, h, w, c0, c1, co):
    """Against torch in 64 bits: FP32 accumulation, one rounding to bf16
    (2^-9 of the value) on output."""
    from seispie_b200 import _lib
    from seispie_b200.engine import check, ptr, stream_handle
    lib, st = _lib.load(), stream_handle(None)
    x0, x1 = _rand(n, h, w, c0, seed=4), _rand(n, h, w, max(c1, 16), seed=5)
    ct = c0 + c1
    wt, b = _rand(9 * co * ct, seed=6), torch.randn(co, device="cuda")
    out = torch.full((n, h, w, co), float("nan"), dtype=torch.bfloat16, device="cuda")
    check(lib.fwi_unet_conv3x3(ptr(x0), c0, ptr(x1) if c1 else None, c1, ptr(wt), ptr(b), co, ptr(out), co, None, 0, n, h,
                               w, 0, st), "conv")
    x = torch.cat([x0, x1[..., :c1]], -1).double().permute(0, 3, 1, 2)
    ref = F.conv2d(x, _torch_w(wt.double(), co, ct), b.double(), padding=1).permute(0, 2, 3, 1)
    scale = float(ref.abs().max())
    assert bool(((out.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-5 * scale).all())


@pytest.mark.parametrize("n,h,w,c", [(1, 2, 2, 8), (3, 10, 14, 24), (2, 6, 130, 256)])
def test_pool_and_upsample_vector_forms(n, h, w, c):
    """The 16-byte forms (aligned buffers) against the scalar forms (buffers
    one element off alignment) on the same values, bit for bit."""
    from seispie_b200 import _lib
    from seispie_b200.engine import check, ptr, stream_handle
    lib, st = _lib.load(), stream_handle(None)

    def off(t):  # the same values two bytes off 16-byte alignment
        o = torch.empty(t.numel() + 1, dtype=t.dtype, device="cuda")[1:].view(t.shape)
        o.copy_(t)
        assert ptr(o) % 16
        return o

    x, small, big = _rand(n, h, w, c, seed=7), _rand(n, h // 2, w // 2, c, seed=8), _rand(n, 2 * h, 2 * w, c, seed=9)
    for name, src, shape, dims in (("pool2", x, small.shape, (n, h, w)), ("up2", x, big.shape, (n, h, w)),
                                   ("up2_bwd", big, x.shape, (n, h, w)), ("pool2_bwd", small, x.shape, (n, h, w, 0)),
                                   ("pool2_bwd", small, x.shape, (n, h, w, 1)), ("relu_bwd", x, x.shape, None)):
        old = _rand(*shape, seed=10)
        outs = []
        for f in (lambda t: t.clone(), off):
            a, o = f(src), f(old)
            if name == "relu_bwd":
                check(lib.fwi_unet_relu_bwd(ptr(o), ptr(a), o.numel(), st), name)
            else:
                check(getattr(lib, "fwi_unet_" + name)(ptr(a), ptr(o), c, *dims, st), name)
            outs.append(o.clone())
        assert torch.equal(outs[0], outs[1]), name
        assert not torch.equal(outs[0], old), name
