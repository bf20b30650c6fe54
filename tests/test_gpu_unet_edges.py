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
