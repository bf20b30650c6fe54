"""The resident steps of small grids (every step of a call in one kernel, a
shot per cluster) against the tiled kernels, bit for bit: at the smallest
grids, at the row counts where the number of rows per thread and of CTAs per
shot changes, with more sources and receivers than are staged, several shots
per wave, odd and even step counts, and a run split between resident and
launched steps."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


NAMES = {"sh": ("vy", "sxy", "szy"), "psv": ("vx", "vz", "sxx", "szz", "sxz")}


def _run(mode, nx, nz, nshots, chunks, npts=7, seed=0):
    from seispie_b200.engine import Grid, ShotBatch, build_model, injection_lists
    rng = np.random.default_rng(seed + 1000 * nx + nz)
    h, dt, nt = 10.0, 1e-3, sum(chunks)
    n = nx * nz
    prm = dict(rho=2600 * (1 + 0.05 * rng.random(n)), lam=8.1e9 * (1 + 0.05 * rng.random(n)),
               mu=8.1e9 * (1 + 0.05 * rng.random(n)))
    m = build_model(mode, Grid(nx, nz, h, h), dt, prm, (3, 0.05, 1, 1, 1, 0))
    src = np.sort(rng.integers(0, n, npts)).astype(np.int32)
    rec = np.concatenate([src, rng.integers(0, n, npts + 3)]).astype(np.int32)
    stf = [torch.as_tensor(rng.standard_normal(npts * nt).astype(np.float32) * 1e6).cuda() for _ in range(3)]
    lib_count = __import__("seispie_b200._lib", fromlist=["load"]).load().fwi_launch_count
    out, launches = [], []
    for disp in (True, False):
        b = ShotBatch(m, nshots, nt, rec, displacement=disp)
        g = torch.Generator(device="cuda").manual_seed(5)
        for k, t in enumerate(b.sig[0] + b.vel[0]):
            scale = 1e6 if k < len(b.sig[0]) else 1.0
            t[..., :nz] = torch.randn(nshots, nx, nz, device="cuda", generator=g) * scale
        d = b.desc(inj=injection_lists(nshots, src, lambda s: -1), stf=stf)
        it, n0 = 0, lib_count()
        for c in chunks:
            b.run(d, False, it, c)
            assert b.cur == (it + c) % 2  # the halves alternate step by step, however the steps were run
            it += c
        launches.append(lib_count() - n0)
        out.append(b)
    return out[0], out[1], launches


def _same(mode, ref, got):
    for c in ((1,) if mode == "sh" else (0, 2)):
        assert torch.equal(ref.traces(c), got.traces(c)), c
    for f in NAMES[mode]:
        assert torch.equal(ref.field(f), got.field(f)), f
    for t in got.sig[got.cur] + got.vel[got.cur]:
        pad = t[..., got.grid.nz:]
        assert pad.numel() == 0 or float(pad.abs().max()) == 0


@pytest.mark.parametrize("mode", ["sh", "psv"])
@pytest.mark.parametrize("nx,nz,nshots,steps", [
    (3, 8, 1, 8), (3, 8, 1, 24), (5, 5, 2, 25), (48, 60, 4, 9), (7, 131, 3, 31), (48, 48, 1, 30), (50, 33, 5, 33), (61, 64, 40, 24),
    (64, 64, 200, 25), (33, 512, 2, 24), (128, 96, 4, 40), (257, 100, 7, 26)])
def test_resident_steps_bit_identical(mode, nx, nz, nshots, steps):
    ref, got, (tiled, resident) = _run(mode, nx, nz, nshots, [steps])
    _same(mode, ref, got)
    assert resident < steps  # these batches take the resident kernel: one launch and the traces' running sums


@pytest.mark.parametrize("mode", ["sh", "psv"])
def test_resident_many_points(mode):
    """More sources and receivers in a CTA's rows than it stages (64)."""
    ref, got, _ = _run(mode, 40, 48, 2, [27], npts=700)
    _same(mode, ref, got)


@pytest.mark.parametrize("mode", ["sh", "psv"])
def test_resident_and_launched_steps_mix(mode):
    """Short calls (launched steps) between long ones (resident)."""
    ref, got, _ = _run(mode, 70, 90, 3, [25, 3, 9, 30, 1, 8])
    _same(mode, ref, got)
