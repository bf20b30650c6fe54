"""Weight gradients at the edges of what the entry points take: scratch that
starts at any float, infinities and NaN beside the image's edges, images
smaller than a pixel tile."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _rand(*shape, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(*shape, device="cuda", generator=g).bfloat16()


def _wgrad(x, g, shift=0):
    """(dw [9, co, c], db [co]) with scratch `shift` floats off its allocation."""
    from seispie_b200 import _lib
    from seispie_b200.engine import check, ptr, stream_handle
    lib, (n, h, w, c), co = _lib.load(), x.shape, g.shape[-1]
    part = torch.full((lib.fwi_unet_wgrad_partials(co, c, n, h, w) + shift,), float("nan"), device="cuda")[shift:]
    dw, db = torch.empty(9, co, c, device="cuda"), torch.empty(co, device="cuda")
    check(lib.fwi_unet_conv3x3_wgrad(ptr(g), co, ptr(x), c, None, 0, n, h, w, ptr(part), ptr(dw), ptr(db),
                                     stream_handle(None)), "wgrad")
    return dw, db


@pytest.mark.parametrize("n,h,w,c,co", [(1, 8, 8, 16, 16), (2, 17, 40, 32, 64), (3, 9, 16, 16, 32), (1, 70, 33, 48, 16)])
def test_scratch_at_any_float(n, h, w, c, co):
    """The scratch holds floats and may start at any of them: the same sums
    whether it is 8-byte aligned or not."""
    x, g = _rand(n, h, w, c, seed=1), _rand(n, h, w, co, seed=2)
    ref = _wgrad(x, g)
    for shift in (1, 2, 3):
        for a, b in zip(ref, _wgrad(x, g, shift)):
            assert torch.equal(a, b)


def _reference(x, g):
    """dw in 64 bits, summed over the pairs of pixels that both lie in the image and over no others."""
    x, g = x.double(), g.double()
    n, h, w, c = x.shape
    dw = torch.zeros(9, g.shape[-1], c, dtype=torch.float64, device=x.device)
    for t in range(9):
        dy, dx = t // 3 - 1, t % 3 - 1
        gy, gx = slice(max(0, -dy), min(h, h - dy)), slice(max(0, -dx), min(w, w - dx))
        xy, xx = slice(max(0, dy), min(h, h + dy)), slice(max(0, dx), min(w, w + dx))
        if h > abs(dy) and w > abs(dx):
            a, b = g[:, gy, gx].reshape(-1, g.shape[-1]), x[:, xy, xx].reshape(-1, c)
            dw[t] = (a[:, :, None] * b[:, None, :]).sum(0)
    return dw


@pytest.mark.parametrize("n,h,w", [(1, 1, 1), (2, 9, 17), (1, 16, 16), (2, 10, 33), (1, 8, 40), (3, 4, 5)])
@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
def test_values_beside_the_edges_meet_no_outside_pixel(n, h, w, value):
    """A non-finite activation in the last row or column reaches the taps that
    pair it with a gradient pixel of the image, and no other tap."""
    for row, col in ((h - 1, 0), (0, w - 1), (h - 1, w - 1)):
        x, g = _rand(n, h, w, 16, seed=3), _rand(n, h, w, 32, seed=4)
        x[0, row, col, 5] = value
        got, ref = _wgrad(x, g)[0].double(), _reference(x, g)
        assert torch.equal(got.isnan(), ref.isnan())
        assert torch.equal(got.isinf() * got.sign(), ref.isinf() * ref.sign())
        ok = ref.isfinite()
        # FP32 sums of exact products, as in the other weight-gradient tests
        assert float((got - ref)[ok].norm()) <= 1e-5 * float(ref[ok].norm()) + 1e-30


# one to eight images per tile, the last tile partly filled, one to more than eight partial sums per weight, 16- and
# 32-column tiles
@pytest.mark.parametrize("n,h,w", [(1, 1, 1), (9, 1, 1), (700, 1, 1), (11, 2, 3), (150, 3, 4), (5, 7, 9), (2, 7, 16),
                                   (3, 1, 20), (40, 3, 33), (3, 4, 33)])
@pytest.mark.parametrize("c,co", [(16, 16), (32, 64)])
def test_small_images(n, h, w, c, co):
    x, g = _rand(n, h, w, c, seed=5), _rand(n, h, w, co, seed=6)
    (dw, db), ref = _wgrad(x, g), _reference(x, g)
    # sums of exact products in FP32: at most their number times 2^-24 of the sum of their sizes
    size = _reference(x.abs(), g.abs())
    assert bool(((dw.double() - ref).abs() <= n * h * w * 2.0 ** -24 * size).all())
    assert float((dw.double() - ref).norm()) <= 1e-5 * float(ref.norm())
    d = db.double() - g.double().sum((0, 1, 2))
    assert bool((d.abs() <= n * h * w * 2.0 ** -24 * g.double().abs().sum((0, 1, 2))).all())


@pytest.mark.parametrize("n,h,w,c", [(300, 2, 2, 8), (1, 70000, 2, 8), (2, 4, 66, 8), (1, 2, 6000, 24), (5, 6, 30, 16)])
def test_rows_of_the_vector_maps(n, h, w, c):
    """Rows shorter than, as long as and longer than a block, more rows than a launch grid: bit for bit against torch
    in FP32 (one rounding of a product with 1/4, or of a sum of four values in the kernels' order)."""
    from seispie_b200 import _lib
    from seispie_b200.engine import check, ptr, stream_handle
    lib, st = _lib.load(), stream_handle(None)
    x, small, big = _rand(n, h, w, c, seed=7), _rand(n, h // 2, w // 2, c, seed=8), _rand(n, 2 * h, 2 * w, c, seed=9)

    def four(t):
        t = t.float()
        return t[:, ::2, ::2] + t[:, ::2, 1::2] + t[:, 1::2, ::2] + t[:, 1::2, 1::2]

    def run(name, src, shape, *more):
        o = torch.full(shape, float("nan"), dtype=torch.bfloat16, device="cuda")
        check(getattr(lib, "fwi_unet_" + name)(ptr(src), ptr(o), c, n, h, w, *more, st), name)
        return o

    twice = lambda t: t.repeat_interleave(2, 1).repeat_interleave(2, 2)  # noqa: E731
    assert torch.equal(run("pool2", x, small.shape), (0.25 * four(x)).bfloat16())
    assert torch.equal(run("up2", x, big.shape), twice(x))
    assert torch.equal(run("up2_bwd", big, x.shape), four(big).bfloat16())
    assert torch.equal(run("pool2_bwd", small, x.shape, 0), (0.25 * twice(small.float())).bfloat16())


# on 148 SMs: 64-pixel tiles by 16, 32 and 64 channels, 128-pixel tiles of three and of five stages by 16, 32 and 64
# channels; images split over two inputs; fewer slices than stages is not possible (nine at least)
@pytest.mark.parametrize("n,h,w,c0,c1,co", [
    (1, 9, 7, 48, 0, 16), (3, 60, 61, 32, 0, 96), (5, 61, 43, 64, 0, 192), (9, 61, 63, 64, 0, 48), (17, 61, 63, 16, 0, 16),
    (16, 61, 63, 64, 32, 32), (5, 61, 63, 32, 0, 32), (9, 61, 63, 64, 64, 64), (9, 61, 63, 16, 16, 64),
    (40, 61, 63, 32, 0, 48)])
def test_convolution_tiles_and_stages(n, h, w, c0, c1, co):
    """Against torch in 64 bits: FP32 accumulation, one rounding to bf16 (2^-9 of the value) on output."""
    import torch.nn.functional as F
    from seispie_b200 import _lib
    from seispie_b200.engine import check, ptr, stream_handle
    lib, st, ct = _lib.load(), stream_handle(None), c0 + c1
    x0, x1, wt = _rand(n, h, w, c0, seed=1), _rand(n, h, w, max(c1, 16), seed=2), _rand(9 * co * ct, seed=3)
    b = torch.randn(co, device="cuda")
    out = torch.full((n, h, w, co), float("nan"), dtype=torch.bfloat16, device="cuda")
    check(lib.fwi_unet_conv3x3(ptr(x0), c0, ptr(x1) if c1 else None, c1, ptr(wt), ptr(b), co, ptr(out), co, None, 0, n,
                               h, w, 0, st), "conv")
    x = torch.cat([x0, x1[..., :c1]], -1).double().permute(0, 3, 1, 2)
    ref = F.conv2d(x, wt.double().view(3, 3, co, ct).permute(2, 3, 0, 1), b.double(), padding=1).permute(0, 2, 3, 1)
    scale = float(ref.abs().max())
    assert bool(((out.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-5 * scale).all())
