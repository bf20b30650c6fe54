"""The row-marching kernel at the edges of its shapes.  Calls of at most seven
steps, or with the ring pinned, are launched one step at a time; every call's
launch count says so here, so that a rule which takes such shapes elsewhere
fails these tests instead of emptying them.  Bit for bit against the tiled
kernels."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

NAMES = {"sh": ("vy", "sxy", "szy"), "psv": ("vx", "vz", "sxx", "szz", "sxz")}


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _march_and_tiled(mode, nx, nz, nshots, chunks=(7, 2), ring=0, cap=0, src=None, rec=None, seed=0):
    from seispie_b200 import _lib
    from seispie_b200.engine import Grid, ShotBatch, build_model, injection_lists
    rng = np.random.default_rng(seed + 1000 * nx + nz)
    n, nt = nx * nz, sum(chunks)
    prm = dict(rho=2600 * (1 + 0.05 * rng.random(n)), lam=8.1e9 * (1 + 0.05 * rng.random(n)),
               mu=8.1e9 * (1 + 0.05 * rng.random(n)))
    m = build_model(mode, Grid(nx, nz, 10.0, 10.0), 1e-3, prm, (3, 0.05, 1, 1, 1, 0))
    if src is None:  # points on consecutive rows, several on one cell
        src = np.sort(rng.integers(0, n, min(n, 7)))
        rec = np.concatenate([src, rng.integers(0, n, 5)])
    src, rec = np.asarray(src, np.int32), np.asarray(rec, np.int32)
    stf = [torch.as_tensor(rng.standard_normal(len(src) * nt).astype(np.float32) * 1e6).cuda() for _ in range(3)]
    count, out = _lib.load().fwi_launch_count, []
    for disp in (True, False):
        b = ShotBatch(m, nshots, nt, rec, displacement=disp)
        if not disp:
            b.ring, b.ctas_per_sm = ring, cap
        g = torch.Generator(device="cuda").manual_seed(5)
        for k, t in enumerate(b.sig[0] + b.vel[0]):
            t[..., :nz] = torch.randn(nshots, nx, nz, device="cuda", generator=g) * (1e6 if k < len(b.sig[0]) else 1.0)
        d = b.desc(inj=injection_lists(nshots, src, lambda s: -1), stf=stf)
        it = 0
        for c in chunks:
            before = count()
            b.run(d, False, it, c)
            assert count() - before == c + (0 if disp else (1 if mode == "sh" else 2))
            it += c
        out.append(b)
    return out


def _same(mode, ref, got):
    for c in ((1,) if mode == "sh" else (0, 2)):
        assert torch.equal(ref.traces(c), got.traces(c)), c
    for f in NAMES[mode]:
        assert torch.equal(ref.field(f), got.field(f)), f
    for h in range(2):
        for t in got.sig[h] + got.vel[h]:
            assert t[..., got.grid.nz:].numel() == 0 or float(t[..., got.grid.nz:].abs().max()) == 0


@pytest.mark.parametrize("mode", ["sh", "psv"])
@pytest.mark.parametrize("nx,nz,nshots", [(1, 8, 2), (2, 5, 1), (3, 4, 3), (4, 129, 1), (5, 128, 2), (7, 132, 2),
                                          (13, 512, 1), (9, 513, 2), (6, 1024, 1), (611, 24, 2), (30, 256, 40)])
def test_shapes(mode, nx, nz, nshots):
    """Few rows and columns, row lengths at the warp and block boundaries, short and long ranges of rows."""
    _same(mode, *_march_and_tiled(mode, nx, nz, nshots))


@pytest.mark.parametrize("mode", ["sh", "psv"])
@pytest.mark.parametrize("ring,cap", [(0, 0), (0, 1), (3, 0), (4, 1), (6, 0), (8, 1)])
def test_many_points(mode, ring, cap):
    """More injection entries and receivers on a row, and in a range of rows,
    than the windows of 128 hold: refilled within a row and between rows."""
    rng = np.random.default_rng(ring)
    nx, nz = 30, 64
    src = np.sort(np.concatenate([rng.integers(4 * nz, 5 * nz, 300), rng.integers(0, nx * nz, 260)]))
    rec = np.concatenate([rng.integers(5 * nz, 6 * nz, 300), rng.integers(0, nx * nz, 260), src[:9]])
    _same(mode, *_march_and_tiled(mode, nx, nz, 40, chunks=(7, 2) if not ring else (11,), ring=ring, cap=cap, src=src,
                                  rec=rec))


def test_row_lengths_in_one_process():
    """A plan for long rows still launches after plans for shorter rows were made, and gives what it gave before."""
    got = []
    for nz in (700, 64, 400, 20, 700):
        ref, b = _march_and_tiled("psv", 20, nz, 1)
        _same("psv", ref, b)
        got.append(b)
    assert torch.equal(got[0].field("sxx"), got[-1].field("sxx"))
