"""The transposed step's injection: entries that share a cell or come in any
order are all summed."""
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


def _model(mode, nx, nz, rng):
    from seispie_b200.engine import Grid, build_model
    n = nx * nz
    base = dict(rho=2600.0, lam=8.1e9, mu=8.1e9)
    if mode == "spin":
        base.update(nu=1.0e9, j=2700.0, mu_c=1.5e8, nu_c=3.0e8)
    prm = {k: v * (1 + 0.05 * rng.random(n)) for k, v in base.items()}
    return build_model(mode, Grid(nx, nz, 10.0, 10.0), 1e-3, prm, (3, 0.05, 1, 1, 1, 0))


@pytest.mark.parametrize("mode", ["sh", "psv", "spin"])
@pytest.mark.parametrize("nshots", [1, 60])
@pytest.mark.parametrize("n", [1, 31, 33, 256, 300])
def test_entries_sharing_cells_in_any_order(mode, nshots, n):
    """One transposed step from a zero state: v~' = sponge dt sum(u~)."""
    from seispie_b200.engine import ShotBatch
    nx, nz, dt = 70, 90, 1e-3
    rng = np.random.default_rng(n)
    m = _model(mode, nx, nz, rng)
    cells = rng.choice(rng.integers(0, nx * nz, 40), n).astype(np.int32)  # many entries a cell, unsorted
    vals = rng.standard_normal((2, nshots * n)).astype(np.float32)
    b = ShotBatch(m, nshots, 1, np.array([5], np.int32))
    stf = [None, None, None]
    for q, c in enumerate(COMPS[mode][:2]):
        stf[c] = torch.as_tensor(vals[q]).cuda()
    inj = (np.arange(nshots + 1, dtype=np.int32) * n, np.tile(cells, nshots), np.arange(nshots * n, dtype=np.int32))
    ks = [torch.zeros((nx, m.grid.pitch), dtype=torch.float64, device="cuda") for _ in range(6 if mode == "spin" else 3)]
    d = b.desc(inj=inj, stf=stf, record=False, kernels=ks)
    z = torch.zeros(1, nshots, nx, m.grid.pitch, device="cuda")
    b.set_segment(d, [z] * NE[mode] + [None] * (6 - NE[mode]), [z if c in COMPS[mode] else None for c in range(3)], 0, 1)
    b.run_transposed(d, 1, 1)
    sponge = m.bound.cpu().numpy()[:, :nz].reshape(-1)
    for q, v in enumerate(b.vel[b.cur][:len(COMPS[mode][:2])]):
        got = v.cpu().numpy()[..., :nz].reshape(nshots, -1)
        for s in range(nshots):
            want, mag = np.zeros(nx * nz), np.zeros(nx * nz)
            np.add.at(want, cells, dt * vals[q, s * n:(s + 1) * n].astype(np.float64))
            np.add.at(mag, cells, dt * np.abs(vals[q, s * n:(s + 1) * n]).astype(np.float64))
            # FP32 sums of at most n terms, dt rounded to FP32, one product with the sponge
            assert np.all(np.abs(got[s] - sponge * want) <= (n + 3) * 2.0 ** -24 * mag)
