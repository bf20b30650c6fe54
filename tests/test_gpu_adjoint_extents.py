"""Transposed steps of grids with more than 65535 tiles along z or x: the
launch grid's second and third extents end there."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

NE = {"sh": 2, "psv": 3, "spin": 6}
COMPS = {"sh": (1,), "psv": (0, 2), "spin": (0, 2, 1)}


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("mode,tile", [("sh", 0), ("psv", 1), ("psv", 0), ("spin", 0)])
@pytest.mark.parametrize("nx,nz", [(3, 32 * 65536 + 17), (20, 32 * 65535)])
def test_many_tiles_along_z(mode, tile, nx, nz):
    """One step from a zero state: v~' = sponge dt u~ at the entries, and zero elsewhere."""
    from seispie_b200 import engine
    from seispie_b200.engine import Grid, ShotBatch, build_model
    n, dt = nx * nz, 1e-3
    prm = dict(rho=np.full(n, 2600.0), lam=np.full(n, 8.1e9), mu=np.full(n, 8.1e9))
    if mode == "spin":
        prm.update({k: np.full(n, v) for k, v in dict(nu=1e9, j=2700.0, mu_c=1.5e8, nu_c=3e8).items()})
    m = build_model(mode, Grid(nx, nz, 10.0, 10.0), dt, prm, (3, 0.05, 1, 1, 1, 0))
    cells = np.array([0, nz // 2, nz - 1, (nx - 1) * nz + 5, n - 40, n - 1], np.int32)
    b = ShotBatch(m, 1, 1, np.array([5], np.int32))
    b.adj_tile = tile
    val = np.arange(1, len(cells) + 1, dtype=np.float32)
    stf = [None, None, None]
    for q, c in enumerate(COMPS[mode][:2]):
        stf[c] = torch.as_tensor(val * (q + 1)).cuda()
    pitch = m.grid.pitch
    ks = [torch.zeros((nx, pitch), dtype=torch.float64, device="cuda") if q not in (2, 5) else None
          for q in range(6 if mode == "spin" else 3)]
    inj = (np.array([0, len(cells)], np.int32), cells, np.arange(len(cells), dtype=np.int32))
    d = b.desc(inj=inj, stf=stf, record=False, kernels=ks)
    z = torch.zeros(1, 1, nx, pitch, device="cuda")
    b.set_segment(d, [z] * NE[mode] + [None] * (6 - NE[mode]), [None] * 3, 0, 1)
    b.run_transposed(d, 1, 1)
    engine.check_device(None, "transposed step")
    sponge = m.bound[:, :nz].reshape(-1).double().cpu().numpy()
    for q, v in enumerate(b.vel[b.cur][:len(COMPS[mode][:2])]):
        got = v[0, :, :nz].reshape(-1)
        assert int((got != 0).sum()) == len(cells)
        # two products of FP32 values, dt rounded to FP32
        want = sponge[cells] * dt * val * (q + 1)
        assert np.all(np.abs(got[torch.as_tensor(cells).long().cuda()].cpu().numpy() - want) <= 4 * 2.0 ** -24 * want)
