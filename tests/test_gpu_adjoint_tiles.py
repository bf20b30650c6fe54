"""The transposed step's tiles of 8, 16, 32 rows and 32 x 64 cells, which the
size of a batch selects: the adjoint fields of a shot have the same bits
whichever tile computes them.  Entries injected into a transposed or a tiled
step that share a cell or come in any order are all summed."""
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


def _fields(m, count, nx, nz, scale, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    t = torch.zeros(count, nx, m.grid.pitch, device="cuda")
    t[..., :nz] = torch.randn(count, nx, nz, device="cuda", generator=g) * scale
    return t


def _run(mode, m, nx, nz, nshots, tile=0, density=True, steps=2):
    """`steps` transposed steps of nshots equal shots."""
    from seispie_b200.engine import ShotBatch, adjoint_injection_lists
    rec = (np.arange(0, nx, 3) * nz + nz // 2).astype(np.int32)
    b = ShotBatch(m, nshots, steps, rec)
    b.adj_tile = tile
    for k, t in enumerate(b.sig[0] + b.vel[0]):
        t.copy_(_fields(m, 1, nx, nz, 1.0, k).expand_as(t))
    seg = [torch.stack([_fields(m, 1, nx, nz, 1e-3, 50 + 7 * q + s).expand(nshots, -1, -1) for s in range(steps)])
           for q in range(NE[mode])] + [None] * (6 - NE[mode])
    ds = [None] * 3
    if density:
        for c in COMPS[mode]:
            ds[c] = torch.stack([_fields(m, 1, nx, nz, 1.0, 90 + 7 * c + s).expand(nshots, -1, -1) for s in range(steps)])
    g = torch.Generator(device="cuda").manual_seed(9)
    one = {c: torch.randn(1, len(rec), steps, device="cuda", generator=g) for c in COMPS[mode] if (mode, c) != ("spin", 1)}
    stf = [one[c].expand(nshots, -1, -1).reshape(-1).contiguous() if c in one else None for c in range(3)]
    ks = [torch.zeros((nx, m.grid.pitch), dtype=torch.float64, device="cuda") if density or q not in (2, 5) else None
          for q in range(6 if mode == "spin" else 3)]
    d = b.desc(inj=adjoint_injection_lists(nshots, rec), stf=stf, record=False, kernels=ks)
    b.set_segment(d, seg, ds, 0, steps)
    b.run_transposed(d, steps, steps)
    from seispie_b200 import engine
    engine.check_device(None, "transposed steps")
    return [t.clone() for t in b.sig[b.cur] + b.vel[b.cur]], ks


@pytest.mark.parametrize("density", [True, False])
@pytest.mark.parametrize("mode,nx,nz,few,many", [
    ("sh", 5, 7, 1, 300), ("sh", 65, 66, 2, 90), ("sh", 33, 131, 1, 90), ("sh", 131, 250, 3, 40),
    ("psv", 5, 7, 1, 300), ("psv", 65, 66, 2, 90), ("psv", 33, 131, 1, 90), ("psv", 130, 403, 1, 8),
    ("psv", 100, 400, 3, 16), ("spin", 5, 7, 1, 300), ("spin", 57, 66, 1, 40), ("spin", 100, 131, 2, 16)])
def test_tiles_by_batch_size_agree(mode, nx, nz, few, many, density):
    rng = np.random.default_rng(nx + nz)
    m = _model(mode, nx, nz, rng)
    f1, k1 = _run(mode, m, nx, nz, few, density=density)
    f2, k2 = _run(mode, m, nx, nz, many, density=density)
    for a, b in zip(f1, f2):
        assert float(a.abs().max()) > 0
        for s in range(many):
            assert torch.equal(a[0], b[s])
    for a, b in zip(k1, k2):
        if a is None:
            continue
        # a per-shot term is summed over the shots of a CTA in FP32 (at most 8 here per 2^-24 each), then in FP64
        scale = float(a.abs().max()) / few
        assert scale > 0 or mode == "sh"
        assert float((a / few - b / many).abs().max()) <= 64 * 2.0 ** -24 * scale
    if mode == "psv":
        f3, _ = _run(mode, m, nx, nz, few, tile=1, density=density)
        for a, b in zip(f1, f3):
            assert torch.equal(a, b)


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


@pytest.mark.parametrize("mode", ["sh", "psv", "spin"])
@pytest.mark.parametrize("n", [1, 33, 300])
def test_sources_sharing_cells_in_any_order(mode, n):
    """One tiled step from a zero state: v = sponge dt/rho sum(stf)."""
    from seispie_b200.engine import ShotBatch
    nx, nz, nshots = 70, 90, 2
    rng = np.random.default_rng(n)
    m = _model(mode, nx, nz, rng)
    cells = rng.choice(rng.integers(0, nx * nz, 40), n).astype(np.int32)
    vals = rng.standard_normal((2, nshots * n)).astype(np.float32)
    b = ShotBatch(m, nshots, 1, np.array([5], np.int32), displacement=True)
    stf = [None, None, None]
    for q, c in enumerate(COMPS[mode][:2]):
        stf[c] = torch.as_tensor(vals[q]).cuda()
    inj = (np.arange(nshots + 1, dtype=np.int32) * n, np.tile(cells, nshots), np.arange(nshots * n, dtype=np.int32))
    b.run(b.desc(inj=inj, stf=stf), False, 0, 1)
    factor = (m.bound * m.buo).cpu().numpy()[:, :nz].reshape(-1).astype(np.float64)
    for q, v in enumerate(b.vel[b.cur][:len(COMPS[mode][:2])]):
        got = v.cpu().numpy()[..., :nz].reshape(nshots, -1)
        for s in range(nshots):
            want, mag = np.zeros(nx * nz), np.zeros(nx * nz)
            np.add.at(want, cells, vals[q, s * n:(s + 1) * n].astype(np.float64))
            np.add.at(mag, cells, np.abs(vals[q, s * n:(s + 1) * n]).astype(np.float64))
            # FP32 sums of at most n terms and three products (one of them in `factor`)
            assert np.all(np.abs(got[s] - factor * want) <= (n + 4) * 2.0 ** -24 * factor * mag)
