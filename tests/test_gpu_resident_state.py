"""What a call of resident steps leaves in the batch's buffers, all of them,
against the launched steps of the row march, bit for bit; the launch count
tells which of the two ran."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _run(mode, nx, nz, nshots, chunks, ring, padding=0.0, npts=5):
    """A batch after len(chunks) calls; ring 0 leaves the choice to the library, 3 asks for the row march."""
    from seispie_b200 import _lib
    from seispie_b200.engine import Grid, ShotBatch, build_model, injection_lists
    rng = np.random.default_rng(1000 * nx + nz)
    n, nt = nx * nz, sum(chunks)
    prm = dict(rho=2600 * (1 + 0.05 * rng.random(n)), lam=8.1e9 * (1 + 0.05 * rng.random(n)),
               mu=8.1e9 * (1 + 0.05 * rng.random(n)))
    m = build_model(mode, Grid(nx, nz, 10.0, 10.0), 1e-3, prm, (3, 0.05, 1, 1, 1, 0))
    src = np.sort(rng.integers(0, n, npts)).astype(np.int32)
    rec = rng.integers(0, n, npts + 2).astype(np.int32)
    stf = [torch.as_tensor(rng.standard_normal(npts * nt).astype(np.float32) * 1e6).cuda() for _ in range(3)]
    b = ShotBatch(m, nshots, nt, rec)
    b.ring = ring
    g = torch.Generator(device="cuda").manual_seed(3)
    for k, t in enumerate(b.sig[0] + b.vel[0]):
        t[..., :nz] = torch.randn(nshots, nx, nz, device="cuda", generator=g) * (1e6 if k < len(b.sig[0]) else 1.0)
        t[..., nz:] = padding
    d = b.desc(inj=injection_lists(nshots, src, lambda s: -1), stf=stf)
    count, it, launches = _lib.load().fwi_launch_count, 0, []
    for c in chunks:
        before = count()
        b.run(d, False, it, c)
        launches.append(count() - before)
        it += c
    ncomp = 1 if mode == "sh" else 2
    for c, l in zip(chunks, launches):  # and a launch per component for the running sums of the traces
        assert l == (1 if ring == 0 and c >= 8 else c) + ncomp
    return b


@pytest.mark.parametrize("mode", ["sh", "psv"])
@pytest.mark.parametrize("nx,nz,nshots", [(3, 6, 2), (50, 33, 3), (128, 96, 2), (61, 130, 1)])
@pytest.mark.parametrize("chunks", [(8,), (9,), (8, 11), (30, 3, 9)])
def test_both_halves(mode, nx, nz, nshots, chunks):
    a, b = _run(mode, nx, nz, nshots, chunks, 3), _run(mode, nx, nz, nshots, chunks, 0)
    assert a.cur == b.cur
    for h in range(2):
        for x, y in zip(a.sig[h] + a.vel[h], b.sig[h] + b.vel[h]):
            assert torch.equal(x, y) and float(x.abs().max()) > 0


@pytest.mark.parametrize("mode", ["sh", "psv"])
@pytest.mark.parametrize("nx,nz,nshots", [(5, 6, 2), (50, 33, 3), (61, 131, 1)])
@pytest.mark.parametrize("padding", [7.0, float("nan"), float("inf")])
def test_row_padding(mode, nx, nz, nshots, padding):
    """Whatever the rows' padding holds before the call, it is zero afterwards and no cell sees it."""
    a, b = _run(mode, nx, nz, nshots, (9,), 3, padding), _run(mode, nx, nz, nshots, (9,), 0, padding)
    clean = _run(mode, nx, nz, nshots, (9,), 0)
    for h in range(2):
        for x, y, z in zip(a.sig[h] + a.vel[h], b.sig[h] + b.vel[h], clean.sig[h] + clean.vel[h]):
            assert torch.equal(y, x) and torch.equal(y, z)
            assert float(y[..., nz:].abs().max()) == 0
    for c in ((1,) if mode == "sh" else (0, 2)):
        assert torch.equal(a.traces(c), b.traces(c))


@pytest.mark.parametrize("mode", ["sh", "psv"])
@pytest.mark.parametrize("nx,nz", [(40, 48), (9, 130)])
def test_many_points(mode, nx, nz):
    """More sources and receivers in a CTA's rows than it stages (64), by the launch count on resident steps."""
    a, b = (_run(mode, nx, nz, 2, (27,), ring, npts=700) for ring in (3, 0))
    for h in range(2):
        for x, y in zip(a.sig[h] + a.vel[h], b.sig[h] + b.vel[h]):
            assert torch.equal(x, y)
    for c in ((1,) if mode == "sh" else (0, 2)):
        assert torch.equal(a.traces(c), b.traces(c)) and float(a.traces(c).abs().max()) > 0
