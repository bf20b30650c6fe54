"""Forward and continuous-adjoint steps with early launches
(fwi_batch.step_overlap = 1) against serialised ones, bit for bit: the row
march alone and with per-step stores, the tiled step of every wave type with
snapshots, the continuous adjoint with its correlation between the steps, and
the multi-instance step.  Calls are short or the ring is pinned where resident
steps, which are one launch, would take them."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

COMPS = {"sh": (1,), "psv": (0, 2), "spin": (0, 2, 1)}


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _model(mode, nx, nz):
    from seispie_b200.engine import Grid, build_model
    rng = np.random.default_rng(nx)
    base = dict(rho=2600.0, lam=8.1e9, mu=8.1e9)
    if mode == "spin":
        base.update(nu=1.0e9, j=2700.0, mu_c=1.5e8, nu_c=3.0e8)
    prm = {k: v * (1 + 0.05 * rng.random(nx * nz)) for k, v in base.items()}
    return build_model(mode, Grid(nx, nz, 10.0, 10.0), 1e-3, prm, (3, 0.05, 1, 1, 1, 0))


def _batch(mode, m, nshots, nt, early, **kw):
    from seispie_b200.engine import ShotBatch, injection_lists
    nx, nz = m.grid.nx, m.grid.nz
    rng = np.random.default_rng(7)
    src = np.sort(rng.integers(0, nx * nz, 9)).astype(np.int32)
    rec = rng.integers(0, nx * nz, 300).astype(np.int32)
    stf = [torch.as_tensor(rng.standard_normal(len(src) * nt).astype(np.float32) * 1e6).cuda() for _ in range(3)]
    b = ShotBatch(m, nshots, nt, rec, **kw)
    b.step_overlap = early
    g = torch.Generator(device="cuda").manual_seed(5)
    for k, t in enumerate(b.sig[0] + b.vel[0]):
        t[..., :nz] = torch.randn(nshots, nx, nz, device="cuda", generator=g) * (1e6 if k < len(b.sig[0]) else 1.0)
    return b, b.desc(inj=injection_lists(nshots, src, lambda s: -1), stf=stf)


def _everything(b):
    return [t for h in range(2) for t in b.sig[h] + b.vel[h]] + b.disp + [
        t for t in list(b.obs) + list(b.snap_u) + list(b.snap_v) if t is not None]


@pytest.mark.parametrize("mode", ["sh", "psv"])
@pytest.mark.parametrize("nx,nz,nshots", [(40, 60, 1), (400, 300, 5), (150, 700, 3)])
@pytest.mark.parametrize("stores", [False, True])
def test_row_march(mode, nx, nz, nshots, stores):
    from seispie_b200 import _lib
    m, nt, out = _model(mode, nx, nz), 20, []
    count = _lib.load().fwi_launch_count
    for early in (0, 1):
        b, d = _batch(mode, m, nshots, nt, early)
        d.ring = 3
        seg = [torch.zeros(nt, nshots, nx, m.grid.pitch, device="cuda") for _ in range(2 if mode == "sh" else 3)]
        ds = [torch.zeros_like(seg[0]) if c in COMPS[mode] else None for c in range(3)]
        if stores:
            b.set_segment(d, seg, ds, 0, nt)
        before = count()
        b.run(d, False, 0, nt)
        assert count() - before == nt + len(COMPS[mode])
        out.append(_everything(b) + (seg + [t for t in ds if t is not None] if stores else []))
    assert all(torch.equal(x, y) and float(x.abs().max()) > 0 for x, y in zip(*out))


@pytest.mark.parametrize("mode", ["sh", "psv", "spin"])
@pytest.mark.parametrize("nx,nz,nshots", [(40, 60, 1), (256, 200, 3), (512, 512, 1)])
def test_tiled_step_and_snapshots(mode, nx, nz, nshots):
    m, nt, sae, out = _model(mode, nx, nz), 24, 4, []
    for early in (0, 1):
        b, d = _batch(mode, m, nshots, nt, early, sae=sae, nsa=nt // sae, snapshots=True, snap_velocity=True)
        b.run(d, False, 0, nt)
        out.append(_everything(b))
    assert all(torch.equal(x, y) for x, y in zip(*out))
    assert all(float(t.abs().max()) > 0 for t in out[0][:4])


@pytest.mark.parametrize("mode", ["sh", "psv"])
@pytest.mark.parametrize("nx,nz,nshots", [(40, 60, 2), (256, 200, 3)])
def test_continuous_adjoint(mode, nx, nz, nshots):
    """The correlation kernel runs between two steps and reads what the next one overwrites."""
    from seispie_b200.engine import adjoint_injection_lists
    m, nt, sae, out = _model(mode, nx, nz), 24, 4, []
    for early in (0, 1):
        b, d = _batch(mode, m, nshots, nt, early, sae=sae, nsa=nt // sae, snapshots=True, snap_velocity=True)
        b.run(d, False, 0, nt)
        g = torch.Generator(device="cuda").manual_seed(2)
        adstf = [torch.randn(nshots * b.nrec * nt, device="cuda", generator=g) if c in COMPS[mode] else None for c in range(3)]
        k = [torch.zeros((nx, m.grid.pitch), dtype=torch.float64, device="cuda") for _ in range(3)]
        b.clear()
        b.run(b.desc(inj=adjoint_injection_lists(nshots, b.rec_cell.cpu().numpy()), stf=adstf, record=False, kernels=k),
              True, 0, nt)
        out.append(_everything(b) + k)
    assert all(torch.equal(x, y) for x, y in zip(*out))
    assert float(out[0][-2].abs().max()) > 0


@pytest.mark.parametrize("sizes,count", [((32, 64), 4), ((64, 160), 12), ((128, 300), 6)])
def test_uneven_instances(sizes, count):
    from seispie_b200.uneven import UnevenBatch, make_instances
    insts, out = make_instances(count, 3, sizes=sizes, nts=(40, 90), shots=(1, 4)), []
    for early in (0, 1):
        ub = UnevenBatch(insts)
        for it in ub.items:
            it[3].step_overlap = early
        ub.prepare()
        ub.clear()
        ub.run()
        torch.cuda.synchronize()
        out.append([t.clone() for _, _, b, _ in ub.items for t in _everything(b)])
    assert all(torch.equal(x, y) for x, y in zip(*out))
