"""The transposed step on every tile that the size of a batch can select (8, 16
or 32 rows by 32 columns, and 32 x 64 cells for P-SV), each named by the rule
itself: the adjoint fields have the same bits on all of them, with more
injected entries than a CTA's list holds (256) and with few, with and without
the density terms, launched early and one by one."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from tests.adjoint_rule import compile_rule  # noqa: E402

NX, NZ, STEPS = 197, 259, 6
NE = {"sh": 2, "psv": 3, "spin": 6}
COMPS = {"sh": (1,), "psv": (0, 2), "spin": (0, 2, 1)}
# shots -> rows, on 148 SMs
BATCHES = {"sh": {1: 8, 2: 16, 8: 32}, "psv": {1: 8, 2: 16, 4: 32, 8: 64}, "spin": {1: 8, 2: 16}}


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    r = compile_rule(str(tmp_path_factory.mktemp("rule")))
    if r is None:
        pytest.skip("no host compiler")
    return r


@pytest.fixture(scope="module")
def models():
    from seispie_b200.engine import Grid, build_model
    rng = np.random.default_rng(1)
    out = {}
    for mode in NE:
        base = dict(rho=2600.0, lam=8.1e9, mu=8.1e9)
        if mode == "spin":
            base.update(nu=1.0e9, j=2700.0, mu_c=1.5e8, nu_c=3.0e8)
        prm = {k: v * (1 + 0.05 * rng.random(NX * NZ)) for k, v in base.items()}
        out[mode] = build_model(mode, Grid(NX, NZ, 10.0, 10.0), 1e-3, prm, (3, 0.05, 1, 1, 1, 0))
    return out


def _run(mode, m, nshots, nrec, density, tile=0, early=1):
    """STEPS transposed steps of nshots equal shots."""
    from seispie_b200 import engine
    from seispie_b200.engine import ShotBatch, adjoint_injection_lists

    def field(seed, scale=1.0):
        g = torch.Generator(device="cuda").manual_seed(seed)
        t = torch.zeros(1, NX, m.grid.pitch, device="cuda")
        t[..., :NZ] = torch.randn(1, NX, NZ, device="cuda", generator=g) * scale
        return t.expand(nshots, -1, -1)

    rec = np.random.default_rng(nrec).integers(0, NX * NZ, nrec).astype(np.int32)
    rec[: nrec // 3] = 40 * NZ + np.arange(nrec // 3) % 70  # several on a cell, many in one tile
    b = ShotBatch(m, nshots, STEPS, rec)
    b.adj_tile, b.step_overlap = tile, early
    for k, t in enumerate(b.sig[0] + b.vel[0]):
        t.copy_(field(k))
    seg = [torch.stack([field(50 + 7 * q + s, 1e-3) for s in range(STEPS)]) for q in range(NE[mode])] + [None] * (6 - NE[mode])
    ds = [torch.stack([field(90 + 7 * c + s) for s in range(STEPS)]) if density and c in COMPS[mode] else None for c in range(3)]
    stf = [None] * 3
    for c in COMPS[mode][:2]:
        g = torch.Generator(device="cuda").manual_seed(9 + c)
        stf[c] = torch.randn(1, nrec, STEPS, device="cuda", generator=g).expand(nshots, -1, -1).reshape(-1).contiguous()
    ks = [torch.zeros((NX, m.grid.pitch), dtype=torch.float64, device="cuda") if density or q not in (2, 5) else None
          for q in range(6 if mode == "spin" else 3)]
    d = b.desc(inj=adjoint_injection_lists(nshots, rec), stf=stf, record=False, kernels=ks)
    b.set_segment(d, seg, ds, 0, STEPS)
    b.run_transposed(d, STEPS, STEPS)
    engine.check_device(None, "transposed steps")
    return b.sig[b.cur] + b.vel[b.cur], ks


@pytest.mark.parametrize("density", [True, False])
@pytest.mark.parametrize("nrec", [40, 300])
@pytest.mark.parametrize("mode", ["sh", "psv", "spin"])
def test_tiles_agree(rule, models, mode, nrec, density):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    ref = None
    runs = [(n, 0) for n in BATCHES[mode]] + ([(3, 1)] if mode == "psv" else [])
    for n, tile in runs:
        if tile == 0 and sms == 148:
            assert rule(mode, NX, NZ, n, sms) == BATCHES[mode][n]
        fields, ks = _run(mode, models[mode], n, nrec, density, tile)
        if ref is None:
            ref = [t[0].clone() for t in fields], [None if k is None else k.clone() for k in ks]
        for a, b in zip(ref[0], fields):
            assert float(a.abs().max()) > 0
            assert all(torch.equal(a, b[s]) for s in range(n))
        for a, k in zip(ref[1], ks):
            if a is not None:
                # a per-shot term is summed over a CTA's shots in FP32 (at most 8 of them), then in FP64
                scale = float(a.abs().max())
                assert scale > 0 or mode == "sh"
                assert float((a - k / n).abs().max()) <= 64 * 2.0 ** -24 * scale


@pytest.mark.parametrize("mode,nshots", [(m, n) for m in BATCHES for n in BATCHES[m]])
def test_early_launches(models, mode, nshots):
    (f0, k0), (f1, k1) = (_run(mode, models[mode], nshots, 60, True, early=e) for e in (0, 1))
    for a, b in zip(f0, f1):
        assert torch.equal(a, b)
    for a, b in zip(k0, k1):
        assert (a is None and b is None) or torch.equal(a, b)
