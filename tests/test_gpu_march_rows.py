"""The row-marching step at the edges of its shapes: grids of a few rows and
columns, row lengths at the warp and block boundaries, every ring depth,
sources and receivers on consecutive rows, and grids of several row lengths
in one process.  Bit for bit against the tiled kernels."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


NAMES = {"sh": ("vy", "sxy", "szy"), "psv": ("vx", "vz", "sxx", "szz", "sxz")}


def _pair(mode, nx, nz, nshots, nt=9, ring=0, cap=0, seed=0):
    """A random state stepped by the tiled and by the row-marching kernels."""
    from seispie_b200.engine import Grid, ShotBatch, build_model, injection_lists
    rng = np.random.default_rng(seed + 1000 * nx + nz)
    h, dt = 10.0, 1e-3
    n = nx * nz
    prm = dict(rho=2600 * (1 + 0.05 * rng.random(n)), lam=8.1e9 * (1 + 0.05 * rng.random(n)),
               mu=8.1e9 * (1 + 0.05 * rng.random(n)))
    m = build_model(mode, Grid(nx, nz, h, h), dt, prm, (3, 0.05, 1, 1, 1, 0))
    # points on consecutive rows, several on one cell
    src = np.sort(rng.integers(0, n, min(n, 7))).astype(np.int32)
    rec = np.concatenate([src, rng.integers(0, n, 5)]).astype(np.int32)
    stf = [torch.as_tensor(rng.standard_normal(len(src) * nt).astype(np.float32) * 1e6).cuda() for _ in range(3)]
    out = []
    for disp in (True, False):
        b = ShotBatch(m, nshots, nt, rec, displacement=disp)
        b.ring, b.ctas_per_sm = (0, 0) if disp else (ring, cap)
        g = torch.Generator(device="cuda").manual_seed(5)
        for k, t in enumerate(b.sig[0] + b.vel[0]):
            scale = 1e6 if k < len(b.sig[0]) else 1.0
            t[..., :nz] = torch.randn(nshots, nx, nz, device="cuda", generator=g) * scale
        d = b.desc(inj=injection_lists(nshots, src, lambda s: -1), stf=stf)
        b.run(d, False, 0, nt)
        out.append(b)
    return out


def _same(mode, ref, got):
    for c in ((1,) if mode == "sh" else (0, 2)):
        assert torch.equal(ref.traces(c), got.traces(c)), c
    for f in NAMES[mode]:
        assert torch.equal(ref.field(f), got.field(f)), f
        pad = got.sig[got.cur][0][..., got.grid.nz:]
        assert pad.numel() == 0 or float(pad.abs().max()) == 0


@pytest.mark.parametrize("mode", ["sh", "psv"])
@pytest.mark.parametrize("nx,nz,nshots", [(1, 8, 2), (2, 5, 1), (3, 4, 3), (4, 129, 1), (5, 128, 2), (7, 132, 2),
                                          (13, 512, 1), (9, 513, 2), (6, 1024, 1), (611, 24, 2), (30, 256, 40)])
def test_grid_shapes(mode, nx, nz, nshots):
    _same(mode, *_pair(mode, nx, nz, nshots))


@pytest.mark.parametrize("mode", ["sh", "psv"])
@pytest.mark.parametrize("ring", [3, 4, 6, 8])
def test_ring_depths(mode, ring):
    """Every ring depth, with one CTA per SM (long ranges) and all that fit."""
    for cap in (0, 1):
        _same(mode, *_pair(mode, 900, 36, 2, ring=ring, cap=cap))


def test_row_lengths_in_one_process():
    """A plan for long rows still launches after plans for shorter rows have
    been made, and gives what it gave before."""
    first = None
    for nz in (700, 64, 400, 20, 700):
        ref, got = _pair("psv", 20, nz, 1)
        _same("psv", ref, got)
        if nz == 700:
            first = first or got
    assert torch.equal(first.field("sxx"), got.field("sxx"))
