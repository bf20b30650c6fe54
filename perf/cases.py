"""The measured cases: the wave-equation work, the gradients and the network
passes that a program built on this package runs, through the entry points
such a program calls.

``listed`` names a dozen cases over the range of grids, batches and options
that the package's own configurations, tests and benchmark use (time axes are
shortened: every step of a run costs the same); ``draw`` gives more of the
same ranges.  ``exact`` evaluates the same maths in plain torch in 64 bits.
"""
import contextlib
import io
import math
import os
import tempfile

import numpy as np
import torch

from seispie_b200 import engine
from seispie_b200.adjoint import AcquisitionSetup, ExactAdjoint, GradientGraph, Seismograms, waveform_misfit
from seispie_b200.engine import Grid, ShotBatch, build_model, injection_lists, point_ids, ricker_stf
from seispie_b200.io import write_model
from seispie_b200.solver import b200
from seispie_b200.unet import LAYERS, UNet
from seispie_b200.uneven import UnevenBatch, make_instances

DEV = "cuda"
# SH and P-SV: 10 m cells, 1.5 ms steps, 20 Hz sources; spin: 1 m cells, 0.15 ms steps, 150 Hz sources
H, DT, F0 = 10.0, 1.5e-3, 20.0
H_SPIN, DT_SPIN, F0_SPIN = 1.0, 1.5e-4, 150.0
ABSORB = (20, 0.015, 1, 1, 1, 0)
SIGMA = 4
SAE = 10
SPIN_BASE = dict(rho=2700.0, lam=8.1e9, mu=8.1e9, nu=1.005e9, j=2700.0, mu_c=1.5e8, nu_c=3.0e8)
COMP = {"sh": (1,), "psv": (0, 2), "spin": (0, 2, 1)}
FIELDS = {"sh": ("sxy", "szy", "vy"), "psv": ("sxx", "szz", "sxz", "vx", "vz"),
          "spin": ("sxx", "szz", "sxz", "syx_c", "syy_c", "syz_c", "vx", "vz", "vy_c")}


def listed():
    return [
        # one SH shot on the smallest configured grid: launch latency
        dict(name="sh_forward_256", kind="forward", mode="sh", nx=256, nz=256, shots=1, nrec=64, nt=200),
        # a modelling run of a few shots on a small, ragged grid
        dict(name="psv_forward_ragged", kind="forward", mode="psv", nx=183, nz=270, shots=3, nrec=37, nt=200),
        # the benchmark's batch: every forward and line-search misfit of its inversions
        dict(name="psv_forward_512", kind="forward", mode="psv", nx=512, nz=512, shots=32, nrec=256, nt=100),
        # the checkerboard inversion's batch (1024 x 512, 64 shots), one column and three rows off the round size
        dict(name="psv_forward_1021", kind="forward", mode="psv", nx=1021, nz=511, shots=64, nrec=256, nt=40),
        # spin forward of a few shots (tiled step, displacement kept)
        dict(name="spin_forward_500", kind="forward", mode="spin", nx=500, nz=412, shots=8, nrec=62, nt=60),
        # the benchmark's exact gradient, replayed from its graphs; a part of the steps stored, the rest recomputed
        dict(name="psv_gradient_512", kind="gradient", mode="psv", nx=512, nz=512, shots=32, nrec=256, nt=120,
             segment=30, tail=45, overlap=True),
        # a small differentiable simulation in a torch program, all of lambda, mu and rho
        dict(name="psv_autograd_128", kind="autograd", mode="psv", nx=128, nz=96, shots=4, nrec=32, nt=150),
        # the plugin's SH gradient from host traces (snapshots every 10 steps, correlated with the adjoint run)
        dict(name="sh_plugin_256", kind="plugin", mode="sh", nx=256, nz=256, shots=16, nrec=64, nt=300),
        # the plugin's P-SV gradient in the geometry the learned preconditioner is trained in, as an optimizer calls it
        dict(name="psv_plugin_256", kind="plugin", mode="psv", nx=256, nz=128, shots=16, nrec=64, nt=300),
        # micropolar-spin gradient with two-level checkpointing
        dict(name="spin_gradient_320", kind="gradient", mode="spin", nx=320, nz=208, shots=4, nrec=40, nt=100,
             segment=0, tail=0, overlap=False),
        # many uneven instances, one graph launch
        dict(name="uneven_12", kind="uneven", count=12, lo=128, hi=384, nt_lo=100, nt_hi=250, shots_hi=8, pick=3),
        # a training step of the preconditioner's network: prediction, loss and parameter gradients
        dict(name="unet_training_8", kind="unet", n=8, h=256, w=128),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["forward"] * 5 + ["gradient"] * 4 + ["autograd"] * 2 + ["plugin"] * 3 + ["uneven", "unet"])
    if kind == "uneven":
        lo = rng.randint(40, 200)
        return dict(kind=kind, count=rng.randint(2, 12), lo=lo, hi=lo + rng.randint(20, 180), nt_lo=rng.randint(60, 100),
                    nt_hi=rng.randint(101, 250), shots_hi=rng.randint(2, 8), pick=rng.randint(0, 10 ** 6))
    if kind == "unet":
        return dict(kind=kind, n=rng.randint(1, 8), h=8 * rng.randint(4, 32), w=8 * rng.randint(4, 16))
    mode = {"forward": ["psv", "psv", "sh", "spin"], "gradient": ["psv", "psv", "sh", "spin"],
            "autograd": ["psv", "sh"], "plugin": ["psv", "sh"]}[kind]
    mode = rng.choice(mode)
    small = kind in ("autograd", "plugin")
    most = 1.2e7 if small else 8e6 if mode == "spin" else 8e8  # cell-updates of one forward sweep
    nx = _log(rng, 48, 256 if small else 1024)
    nz = _log(rng, 44, 256 if small else 1024)
    if kind == "forward" and rng.random() < 0.1:
        nx, nz = _log(rng, 48, 300), rng.randint(1025, 1400)  # deeper than the row-marching step takes
    shots = _log(rng, 1, 16 if small else 64)
    nt = rng.randint(60, 300 if small else 160)
    while shots > 1 and nx * nz * shots * nt > (most if kind != "gradient" else most / 3):
        shots = (shots + 1) // 2
    c = dict(kind=kind, mode=mode, nx=nx, nz=nz, shots=shots, nrec=rng.randint(4, max(5, min(nx, 256) - 2)), nt=nt)
    if kind == "gradient":
        seg = 0 if mode == "spin" else rng.randint(8, 40)
        c.update(segment=seg, tail=0 if mode == "spin" else rng.randint(0, nt // 2),
                 overlap=mode != "spin" and rng.random() < 0.7)
    if kind == "plugin":
        c["nt"] = nt - nt % SAE
    return c


# ------------------------------------------------------------------ inputs

def _axes(case):
    spin = case["mode"] == "spin"
    return (H_SPIN, DT_SPIN, F0_SPIN) if spin else (H, DT, F0)


def _rng(seed, salt=0):
    return np.random.default_rng([int(seed), salt])


def _board(rng, nx, nz):
    """A checkerboard on a smooth background, in [-1, 1]."""
    i, j = np.arange(nx)[:, None], np.arange(nz)[None, :]
    sq, oi, oj = int(rng.integers(16, 49)), int(rng.integers(0, 16)), int(rng.integers(0, 16))
    board = np.where((((i + oi) // sq) + ((j + oj) // sq)) % 2 == 0, 1.0, -1.0)
    smooth = np.sin(rng.uniform(1, 6) * i / nx + rng.uniform(0, 6)) * np.cos(rng.uniform(1, 6) * j / nz)
    return 0.6 * board + 0.4 * smooth


def _params(case, rng):
    nx, nz = case["nx"], case["nz"]
    b = _board(rng, nx, nz).ravel()
    if case["mode"] == "spin":
        return {k: (v * (1 + 0.04 * b * (1 if k != "rho" else -1))).astype(np.float32) for k, v in SPIN_BASE.items()}
    vp = (3000.0 * (1 + 0.05 * b)).astype(np.float32)
    return dict(vp=vp, vs=(vp / np.sqrt(3.0)).astype(np.float32), rho=(2600.0 * (1 + 0.03 * b)).astype(np.float32))


def _points(case, rng):
    """One source per shot and the receiver line, on cells, near the surface."""
    h, dt, f0 = _axes(case)
    nx, nz, ns, nr = case["nx"], case["nz"], case["shots"], case["nrec"]
    depth = int(rng.integers(8, 13))
    src = np.array([[min(nx - 4, max(4, int((s + rng.uniform(0.2, 0.8)) * nx / ns))) * h, depth * h, 0, f0, 1.2 / f0,
                     rng.uniform(-60, 60), 1e10] for s in range(ns)])
    rec = np.array([[int((r + 0.5) * nx / nr) * h, (depth + 3) * h] for r in range(nr)])
    return src, rec


def _arrivals(case, rng, src, rec):
    """Observed traces [shot, receiver, t]: a wavelet per shot with a hyperbolic
    moveout, of the amplitude the simulated displacements have."""
    h, dt, f0 = _axes(case)
    nt = case["nt"]
    amp = 0.06 if case["mode"] == "spin" else 5.0
    t = np.arange(nt) * dt
    off = (src[:, None, 0] - rec[None, :, 0]) * rng.uniform(0.9, 1.1)
    t0 = 1.2 / f0 + np.sqrt(off ** 2 + (20 * h) ** 2) / 2500.0
    a = (math.pi * f0) ** 2 * (t[None, None] - t0[..., None]) ** 2
    g = (1 - 2 * a) * np.exp(-a) / np.sqrt(1 + np.abs(off) / (10 * h))[..., None]
    return (amp * rng.uniform(0.5, 1.5) * g).astype(np.float32)


def _ids(case, pts):
    h = np.float32(_axes(case)[0])
    return point_ids(pts, h, h, case["nz"])


def _wave_inputs(case, seed):
    rng = _rng(seed)
    prm = _params(case, rng)
    src, rec = _points(case, rng)
    data = {c: _arrivals(case, rng, src, rec) for c in ((1,) if case["mode"] == "sh" else (0, 2))}
    return prm, src, rec, data


def _model(case, prm):
    h, dt, _ = _axes(case)
    return build_model(case["mode"], Grid(case["nx"], case["nz"], h, h), dt, prm, ABSORB, DEV)


def _instances(case, seed):
    # the shapes belong to the case, the models to the seed
    insts = make_instances(case["count"], seed=case["pick"], sizes=(case["lo"], case["hi"]),
                           nts=(case["nt_lo"], case["nt_hi"]), shots=(2, case["shots_hi"]))
    for k, i in enumerate(insts):
        rng = _rng(seed, k + 1)
        b = _board(rng, i.nx, i.nz).ravel()
        vp = (3000.0 * (1 + 0.05 * b)).astype(np.float32)
        i.params = dict(vp=vp, vs=(vp / np.sqrt(3.0)).astype(np.float32),
                        rho=(2600.0 * (1 + 0.03 * b)).astype(np.float32))
        i.dt = DT
        i.src[:, 3], i.src[:, 4] = F0, 1.2 / F0
    return insts


def _planes(case, seed):
    """Network input (gradient, illumination and model planes) and target."""
    n, h, w = case["n"], case["h"], case["w"]
    rng = _rng(seed)
    i, j = np.linspace(0, 1, h)[:, None], np.linspace(0, 1, w)[None, :]
    x = np.zeros((n, 3, h, w), np.float32)
    y = np.zeros((n, h, w), np.float32)
    for q in range(n):
        b = _board(rng, h, w)
        g = sum(rng.uniform(-1, 1) * np.sin(rng.uniform(2, 40) * i + rng.uniform(0, 6)) * np.cos(rng.uniform(2, 40) * j)
                for _ in range(4))
        x[q, 0] = g / np.abs(g).max()
        x[q, 1] = np.clip(1 - 0.8 * j + 0.1 * np.sin(9 * i), 0, 1)
        x[q, 2] = 0.05 * b
        y[q] = 0.7 * b - 0.3 * x[q, 0]
    return x, y


def _weights_of(net, seed):
    """Seeded weights with biases, as after some training."""
    w = net.w.cpu().numpy().copy()
    rng = _rng(seed, 77)
    for name, _, _, co in LAYERS:
        o, _ = net.offsets[name + ".b"]
        w[o:o + co] = 0.05 * rng.standard_normal(co)
    return w


# ------------------------------------------------------------------ prepare and run

class _Plan:
    """What a program keeps between calls, by name."""

    def __init__(self, **kw):
        self.__dict__.update(kw)


def _solver(case, prm, src, rec, data):
    """The solver plugin as the runner sets it up, from files in a temporary
    directory (read once here)."""
    h, dt, _ = _axes(case)
    sh = case["mode"] == "sh"
    with tempfile.TemporaryDirectory() as root:
        write_model(os.path.join(root, "model"), case["nx"], case["nz"], h, h, prm)
        np.savetxt(os.path.join(root, "sources.dat"), src)
        np.savetxt(os.path.join(root, "stations.dat"), rec)
        for c, arr in data.items():
            for s in range(case["shots"]):
                arr[s].tofile(os.path.join(root, "v%s_%06d.npy" % ("xyz"[c], s)))
        s = b200()
        s.config = dict(nt=str(case["nt"]), dt=repr(dt), sh="yes" if sh else "no", psv="no" if sh else "yes",
                        abs_width=str(ABSORB[0]), abs_alpha=repr(ABSORB[1]), abs_left="yes", abs_right="yes",
                        abs_bottom="yes", abs_top="no", save_coordinates="", save_snapshot="0",
                        combine_sources="no", adjoint_interval=str(SAE), smooth=str(SIGMA), threads_per_block="256")
        s.path = dict(model_true=os.path.join(root, "model"), model_init=os.path.join(root, "model"),
                      sources=os.path.join(root, "sources.dat"), stations=os.path.join(root, "stations.dat"),
                      output=root, traces=root)
        s.mpi = None
        s.setup(None)
        s.import_model(0)
        s.import_sources()
        s.import_stations()
        s.import_traces()
    return s


_planned = set()


def _plan_rows():
    """The launch plans of the forward step for every row length, once per
    process and in ascending order, as a program that works with grids of
    several depths in one process has to make them: a plan for shorter rows
    made after one for longer rows withdraws the shared memory that the
    longer rows' plan needs."""
    if _planned:
        return
    _planned.add(True)
    for nz in range(128, 1025, 128):
        for mode in ("sh", "psv"):
            case = dict(mode=mode, nx=8, nz=nz, shots=1, nrec=1, nt=1)
            rng = _rng(0)
            b = ShotBatch(_model(case, _params(case, rng)), 1, 1, _ids(case, _points(case, rng)[1]))
            b.run(b.desc(), False, 0, 1)


def prepare(case, seed):
    kind = case["kind"]
    _plan_rows()
    if kind == "unet":
        x, y = _planes(case, seed)
        net = UNet(DEV, seed=seed % 1000)
        net.load_flat(_weights_of(net, seed))
        return _Plan(case=case, net=net, x=torch.as_tensor(x, device=DEV), y=torch.as_tensor(y, device=DEV))
    if kind == "uneven":
        ub = UnevenBatch(_instances(case, seed))
        ub.capture()
        return _Plan(case=case, batch=ub)
    prm, src, rec, data = _wave_inputs(case, seed)
    if kind == "plugin":
        return _Plan(case=case, solver=_solver(case, prm, src, rec, data))
    h, dt, _ = _axes(case)
    nt, ns = case["nt"], case["shots"]
    if kind == "autograd":
        setup = AcquisitionSetup(case["mode"], Grid(case["nx"], case["nz"], h, h), dt, nt, src, rec, ABSORB)
        vp, vs, rho = (torch.as_tensor(prm[k], device=DEV).view(case["nx"], case["nz"]) for k in ("vp", "vs", "rho"))
        obs = torch.stack([torch.as_tensor(data[c], device=DEV) for c in sorted(data)])
        return _Plan(case=case, setup=setup, lam=(rho * (vp * vp - 2 * vs * vs)).contiguous(),
                     mu=(rho * vs * vs).contiguous(), rho=rho.contiguous(), obs=obs)
    m = _model(case, prm)
    sid, rid = _ids(case, src), _ids(case, rec)
    stf, _ = ricker_stf(src, nt, dt, DEV)
    if kind == "forward":
        b = ShotBatch(m, ns, nt, rid)
        return _Plan(case=case, batch=b, desc=b.desc(inj=injection_lists(ns, sid, lambda s: s), stf=stf), stf=stf)
    per_step = 3 * 4 * ns * case["nx"] * m.grid.pitch if case["mode"] == "psv" else 2 * 4 * ns * case["nx"] * m.grid.pitch
    ea = ExactAdjoint(m, nt, sid, lambda s: s, ns, stf, rid, segment=case["segment"] or None,
                      levels=2 if case["mode"] == "spin" else 1, tail_memory=case["tail"] * per_step,
                      overlap=case["overlap"], density=case["mode"] == "spin")
    obs = {c: torch.as_tensor(data[c], device=DEV).reshape(-1) for c in data}

    def between(tr):
        grads, mis = [None, None, None], []
        for c in obs:
            g = torch.empty(ns * len(rid) * nt, dtype=torch.float32, device=DEV)
            mis.append(engine.misfit_tracegrad(obs[c], tr[c].reshape(-1).contiguous(), g, ns, len(rid), nt, dt))
            grads[c] = g.view(ns, len(rid), nt)
        return grads, mis

    # spin batches are too large to keep their graphs and are launched step by step
    graph = GradientGraph(ea, between) if case["mode"] != "spin" else None
    return _Plan(case=case, ea=ea, between=between, graph=graph, stf=stf)


def run(state):
    case = state.case
    kind = case["kind"]
    if kind == "forward":
        b = state.batch
        b.clear()
        b.run(state.desc, False, 0, b.nt)
        return {"traces": [b.traces(c) for c in COMP[case["mode"]]],
                "state": [b.field(f) for f in FIELDS[case["mode"]]]}
    if kind == "gradient":
        if state.graph is not None:
            tr, mis, ks = state.graph.replay()
        else:
            tr = state.ea.forward()
            g, mis = state.between(tr)
            ks = state.ea.backward(g)
        grid = state.ea.model.grid
        smoothed = [engine.smooth(k, grid, SIGMA) for q, k in enumerate(ks)
                    if k is not None and not (case["mode"] == "sh" and q == 0)]
        misfit = sum(float(m.sum().item()) for m in mis)
        return {"traces": [tr[c] for c in COMP[case["mode"]]], "misfit": misfit, "gradients": smoothed}
    if kind == "autograd":
        lam, mu, rho = (t.clone().requires_grad_() for t in (state.lam, state.mu, state.rho))
        tr = Seismograms.apply(lam, mu, rho, state.setup)
        loss = waveform_misfit(tr, state.obs, state.setup.dt)
        loss.backward()
        grads = [mu.grad, rho.grad] if case["mode"] == "sh" else [lam.grad, mu.grad, rho.grad]
        return {"traces": tr.detach(), "loss": float(loss.item()), "gradients": grads}
    if kind == "plugin":
        with contextlib.redirect_stdout(io.StringIO()):  # the solver reports its progress
            if case["mode"] == "sh":
                k, misfit, mu = state.solver.compute_gradient()
            else:
                k, misfit, mu = state.solver.compute_gradient_device()
        return {"gradient": k, "misfit": misfit, "mu": mu}
    if kind == "uneven":
        state.batch.graph.replay()
        return [[t for t in state.batch.traces(k) if t is not None] for k in range(case["count"])]
    net = state.net
    out = net.forward(state.x)
    loss, gout = net.mse(out, state.y)
    net.backward(gout)
    return {"out": out, "loss": float(loss.item()), "gradients": {k: net.view(k, net.g) for k in net.offsets}}


# ------------------------------------------------------------------ work

# arithmetic of one cell-update (stencils of 4 taps: two differences, two products, one difference)
FLOPS = {"sh": 36, "psv": 80, "spin": 160}
MODEL = {"sh": 3, "psv": 4, "spin": 7}  # model fields a step reads


def _sweep(mode, nx, nz, shots, nrec, nt):
    """(bytes, flops) of one forward sweep: the model, the wavelets and nothing
    else go in, the traces come out."""
    return (4.0 * (MODEL[mode] * nx * nz + len(COMP[mode]) * shots * nt * (1 + nrec)),
            float(FLOPS[mode]) * nx * nz * shots * nt)


def work(case):
    kind = case["kind"]
    if kind == "unet":
        px = float(case["n"] * case["h"] * case["w"])
        fl, par = 0.0, 0
        level = {"e1": 0, "d1": 0, "e2": 1, "d2": 1, "e3": 2, "d3": 2, "ba": 3, "bb": 3}
        for name, c0, c1, co in LAYERS:
            one = 2.0 * px / 4 ** level[name[:2]] * 9 * (c0 + c1) * co
            fl += one * (2 if name == "e1a" else 3)
            par += 9 * (c0 + c1) * co + co
        return {"bytes": 4.0 * (5 * px + 2 * par), "flops": fl}
    if kind == "uneven":
        by = fl = 0.0
        for i in _instances(case, 0):
            b, f = _sweep(i.mode, i.nx, i.nz, len(i.src), len(i.rec), i.nt)
            by, fl = by + b, fl + f
        return {"bytes": by, "flops": fl}
    mode, cells = case["mode"], case["nx"] * case["nz"]
    by, fl = _sweep(mode, cells, 1, case["shots"], case["nrec"], case["nt"])
    if kind == "forward":
        by += 4.0 * len(FIELDS[mode]) * cells * case["shots"]
        return {"bytes": by, "flops": fl}
    # gradients: the observed traces go in, the kernels come out, the adjoint costs what the forward does
    by += 4.0 * len(COMP[mode]) * case["shots"] * case["nt"] * case["nrec"] + 4.0 * MODEL[mode] * cells
    return {"bytes": by, "flops": 2 * fl}


# ------------------------------------------------------------------ 64-bit values

F64 = torch.float64


def _dm(f, ax, h):
    """D- along axis ax (-2: x, -1: z): zero unless 2 <= i < n-2."""
    n = f.shape[ax]
    s = lambda a, b: f.narrow(ax, a, b - a)  # noqa: E731
    d = 9 / (8 * h) * (s(2, n - 2) - s(1, n - 3)) - 1 / (24 * h) * (s(3, n - 1) - s(0, n - 4))
    return torch.nn.functional.pad(d, (0, 0, 2, 2) if ax == -2 else (2, 2))


def _dp(f, ax, h):
    """D+ along axis ax: zero unless 1 <= i < n-2."""
    n = f.shape[ax]
    s = lambda a, b: f.narrow(ax, a, b - a)  # noqa: E731
    d = 9 / (8 * h) * (s(2, n - 1) - s(1, n - 2)) - 1 / (24 * h) * (s(3, n) - s(0, n - 3))
    return torch.nn.functional.pad(d, (0, 0, 1, 2) if ax == -2 else (1, 2))


def _sponge(nx, nz):
    w, a, left, right, bottom, top = ABSORB
    x, z = np.ones(nx), np.ones(nz)
    for i in range(nx):
        if left and i + 1 < w:
            x[i] *= math.exp(-(a * (w - i - 1)) ** 2)
        if right and i > nx - w:
            x[i] *= math.exp(-(a * (w + i - nx)) ** 2)
    for j in range(nz):
        if bottom and j > nz - w:
            z[j] *= math.exp(-(a * (w + j - nz)) ** 2)
        if top and j + 1 < w:
            z[j] *= math.exp(-(a * (w - j - 1)) ** 2)
    return torch.as_tensor(x[:, None] * z[None, :], device=DEV)


def _ricker(src, nt, dt):
    """[component x, y, z][source, t]."""
    t = np.arange(nt) * dt
    out = np.zeros((3, len(src), nt))
    for q, s in enumerate(src):
        a = (math.pi * s[3]) ** 2
        w = -s[6] * (1 - 2 * a * (t - s[4]) ** 2) * np.exp(-a * (t - s[4]) ** 2)
        ang = math.radians(s[5])
        out[:, q] = w * math.sin(ang), w, -w * math.cos(ang)
    return torch.as_tensor(out, device=DEV)


def _simulate(mode, h, dt, nt, prm, bound, stf, sxz, rxz, each=None):
    """Steps of the shots of stf; returns ([trace per component], [state]).
    ``each(it, u)``, if given, sees the displacement before step it."""
    ns, (nx, nz) = stf.shape[1], bound.shape
    z = torch.zeros((ns, nx, nz), dtype=F64, device=DEV)
    nv = {"sh": 1, "psv": 2, "spin": 3}[mode]
    sig = [z] * {"sh": 2, "psv": 3, "spin": 6}[mode]
    v, u = [z] * nv, [z] * nv
    shot = torch.arange(ns, device=DEV)
    buo = dt / prm["rho"]
    lam, mu = prm.get("lam"), prm["mu"]
    put = lambda f, val: f.index_put((shot, sxz[0], sxz[1]), val, accumulate=True)  # noqa: E731
    rec = []
    for it in range(nt):
        if each is not None:
            each(it, u)
        if mode == "sh":
            d = [put(_dm(sig[0], -2, h) + _dm(sig[1], -1, h), stf[1][:, it])]
        else:
            d = [_dm(sig[0], -2, h) + _dm(sig[2], -1, h), _dm(sig[2], -2, h) + _dm(sig[1], -1, h)]
            if mode == "spin":
                d = [d[0] + _dm(sig[4], -1, h), d[1] - _dm(sig[4], -2, h),
                     _dm(sig[3], -2, h) + _dm(sig[5], -1, h) + 2 * sig[4]]
            d = [put(d[0], stf[0][:, it]), put(d[1], stf[2][:, it])] + d[2:]
        v = [bound * (a + (dt / prm["j"] if q == 2 else buo) * b) for q, (a, b) in enumerate(zip(v, d))]
        if each is not None:
            u = [a + dt * b for a, b in zip(u, v)]
        rec.append(torch.stack([a[:, rxz[0], rxz[1]] for a in v]))
        if mode == "sh":
            sig = [sig[0] + dt * mu * _dp(v[0], -2, h), sig[1] + dt * mu * _dp(v[0], -1, h)]
            continue
        xx, xz, zx, zz = _dp(v[0], -2, h), _dp(v[0], -1, h), _dp(v[1], -2, h), _dp(v[1], -1, h)
        l2m = lam + 2 * mu
        new = [sig[0] + dt * (l2m * xx + lam * zz), sig[1] + dt * (l2m * zz + lam * xx), sig[2] + dt * mu * (xz + zx)]
        if mode == "spin":
            mnc = prm["mnc"]
            new += [sig[3] + dt * mnc * _dp(v[2], -2, h), sig[4] + 2 * dt * prm["nu"] * (-v[2] - 0.5 * (zx - xz)),
                    sig[5] + dt * mnc * _dp(v[2], -1, h)]
        sig = new
    tr = torch.cumsum(torch.stack(rec, -1), -1) * dt  # [component, shot, receiver, t]
    return list(tr), sig + v


def _params64(mode, prm, nx, nz):
    t = {k: torch.as_tensor(np.asarray(a, np.float64), device=DEV).view(nx, nz) for k, a in prm.items()}
    if mode == "spin":
        t["mnc"] = t["mu_c"] + t["nu_c"]
    else:
        t["mu"] = t["rho"] * t["vs"] ** 2
        t["lam"] = t["rho"] * (t["vp"] ** 2 - 2 * t["vs"] ** 2)
    return t


def _cells(pts, h):
    i = np.rint(pts[:, :2] / h).astype(np.int64)
    return torch.as_tensor(i[:, 0], device=DEV), torch.as_tensor(i[:, 1], device=DEV)


def _taper(nt, dt):
    t, end = np.arange(nt) * dt, (nt - 1) * dt
    tw = end / 10
    w = np.ones(nt)
    lo, hi = t <= tw, t >= end - tw
    w[lo] = 0.5 + 0.5 * np.cos(math.pi * (tw - t[lo]) / tw)
    w[hi] = 0.5 + 0.5 * np.cos(math.pi * (end - tw - t[hi]) / tw)
    return torch.as_tensor(w, device=DEV)


def _smooth64(k):
    """Gaussian smoothing, normalised by the mass inside the grid; [nx*nz]."""
    def mat(n):
        d = torch.arange(n, device=DEV, dtype=F64)
        w = torch.exp(-(d[:, None] - d[None, :]) ** 2 / (2.0 * SIGMA ** 2))
        return w / w.sum(1, keepdim=True)
    return (mat(k.shape[0]) @ k @ mat(k.shape[1]).T).reshape(-1)


def _exact_gradient(case, prm, src, rec, data, names, unit):
    """(traces, loss, norms, {name: dloss/dname}) with loss the tapered squared
    residual and norms the per-shot, per-component norms; a few shots at a time."""
    mode, nx, nz, nt = case["mode"], case["nx"], case["nz"], case["nt"]
    h, dt, _ = _axes(case)
    p = _params64(mode, prm, nx, nz)
    p["buo"] = dt / p["rho"]
    if mode == "spin":
        p["buo_j"] = dt / p["j"]
    for n in names:
        p[n] = p[n].detach().requires_grad_()
    q = dict(p)
    if "buo" in names:
        q["rho"] = dt / p["buo"]
    if "buo_j" in names:
        q["j"] = dt / p["buo_j"]
    stf, bound = _ricker(src, nt, dt), _sponge(nx, nz)
    sx, sz = _cells(src, h)
    rxz = _cells(rec, h)
    w = _taper(nt, dt)
    per = max(1, int(2.5e10 / (8.0 * nx * nz * nt * (10 if mode != "spin" else 24))))
    traces, loss, norm = [], 0.0, 0.0
    grads = {n: 0.0 for n in names}
    for s0 in range(0, case["shots"], per):
        s = slice(s0, min(case["shots"], s0 + per))
        tr, _ = _simulate(mode, h, dt, nt, q, bound, stf[:, s], (sx[s], sz[s]), rxz)
        part = 0.0
        for c, t in zip(COMP[mode], tr):
            if c in data:
                r = (t - torch.as_tensor(data[c][s], device=DEV).double()) * w
                part = part + (r * r).sum()
                norm += float((r.detach() ** 2).sum((1, 2)).sqrt().sum())
        loss += float(part.detach())
        for n, g in zip(names, torch.autograd.grad(part, [p[n] for n in names], allow_unused=True)):
            grads[n] = grads[n] + (unit * g if g is not None else torch.zeros_like(p[n]))
        traces.append([t.detach() for t in tr])
        del tr, part
    return [torch.cat(t) for t in zip(*traces)], loss, norm, grads


def _exact_sh_reference(case, prm, src, rec, data):
    """The snapshot-correlation gradient: displacement kept every SAE steps,
    the residual run back as sources at the receivers, D+ u_adj . D+ u_fwd
    summed with SAE*dt; (smoothed kernel, misfit)."""
    nx, nz, nt, ns = case["nx"], case["nz"], case["nt"], case["shots"]
    h, dt, _ = _axes(case)
    p = _params64("sh", prm, nx, nz)
    bound, nsa, snaps = _sponge(nx, nz), nt // SAE, {}

    def keep(it, u):
        if (it + 1) % SAE == 0:
            snaps[nsa - (it + 1) // SAE] = u[0]

    tr, _ = _simulate("sh", h, dt, nt, p, bound, _ricker(src, nt, dt), _cells(src, h), _cells(rec, h), keep)
    w = _taper(nt, dt)
    r = (torch.as_tensor(data[1], device=DEV).double() - tr[0]) * w
    misfit = float((r * r).sum((1, 2)).sqrt().sum())
    ad = (2 * r * w).flip(-1)
    z = torch.zeros((ns, nx, nz), dtype=F64, device=DEV)
    sxy, szy, v, u, k = z, z, z, z, torch.zeros((nx, nz), dtype=F64, device=DEV)
    rx, rz = _cells(rec, h)
    buo, mu = dt / p["rho"], p["mu"]
    for it in range(nt):
        d = _dm(sxy, -2, h) + _dm(szy, -1, h)
        d[:, rx, rz] += ad[..., it]
        v = bound * (v + buo * d)
        u = u + dt * v
        sxy, szy = sxy + dt * mu * _dp(v, -2, h), szy + dt * mu * _dp(v, -1, h)
        if it % SAE == 0:
            f = snaps[it // SAE]
            k += ((_dp(u, -2, h) * _dp(f, -2, h) + _dp(u, -1, h) * _dp(f, -1, h)) * (SAE * dt)).sum(0)
    return _smooth64(k), misfit


def _exact_unet(case, seed):
    """The network on its bf16 weights, in 64 bits."""
    F = torch.nn.functional
    x, y = _planes(case, seed)
    net = UNet(DEV, seed=seed % 1000)
    w = _weights_of(net, seed)
    par = {}
    for name, (o, shape) in net.offsets.items():
        t = torch.as_tensor(w[o:o + int(np.prod(shape))], device=DEV).view(shape)
        if name.endswith(".w") and name != "head.w":
            t = t.bfloat16()
        par[name] = t.double().requires_grad_()

    def conv(name, t):
        k = par[name + ".w"]
        return F.relu(F.conv2d(t, k.view(3, 3, k.shape[1], k.shape[2]).permute(2, 3, 0, 1), par[name + ".b"], padding=1))

    t = F.pad(torch.as_tensor(x, device=DEV).bfloat16().double(), (0, 0, 0, 0, 0, 13))
    skip = []
    for a, b in (("e1a", "e1b"), ("e2a", "e2b"), ("e3a", "e3b"), ("ba", "bb")):
        t = conv(b, conv(a, t if a == "e1a" else F.avg_pool2d(t, 2)))
        skip.append(t)
    skip.pop()
    for a, b in (("d3a", "d3b"), ("d2a", "d2b"), ("d1a", "d1b")):
        t = conv(b, conv(a, torch.cat([F.interpolate(t, scale_factor=2, mode="nearest"), skip.pop()], 1)))
    out = (t * par["head.w"].view(1, 16, 1, 1)).sum(1) + par["head.b"]
    loss = ((out - torch.as_tensor(y, device=DEV).double()) ** 2).mean()
    grads = dict(zip(par, torch.autograd.grad(loss, list(par.values()))))
    return {"out": out.detach(), "loss": float(loss.detach()), "gradients": grads}


def exact(case, seed):
    kind = case["kind"]
    if kind == "unet":
        return _exact_unet(case, seed)
    if kind == "uneven":
        out = []
        with torch.no_grad():
            for i in _instances(case, seed):
                p = _params64(i.mode, i.params, i.nx, i.nz)
                tr, _ = _simulate(i.mode, i.h, i.dt, i.nt, p, _sponge(i.nx, i.nz), _ricker(i.src, i.nt, i.dt),
                                  _cells(i.src, i.h), _cells(i.rec, i.h))
                out.append(tr)
        return out
    prm, src, rec, data = _wave_inputs(case, seed)
    mode, nx, nz, nt = case["mode"], case["nx"], case["nz"], case["nt"]
    h, dt, _ = _axes(case)
    if kind == "forward":
        p, bound, stf = _params64(mode, prm, nx, nz), _sponge(nx, nz), _ricker(src, nt, dt)
        sx, sz = _cells(src, h)
        parts = []
        with torch.no_grad():
            for s0 in range(0, case["shots"], 16):
                s = slice(s0, s0 + 16)
                parts.append(_simulate(mode, h, dt, nt, p, bound, stf[:, s], (sx[s], sz[s]), _cells(rec, h)))
        return {"traces": [torch.cat(t) for t in zip(*(a for a, _ in parts))],
                "state": [torch.cat(t) for t in zip(*(b for _, b in parts))]}
    if kind == "plugin" and mode == "sh":
        with torch.no_grad():
            k, misfit = _exact_sh_reference(case, prm, src, rec, data)
        return {"gradient": k, "misfit": misfit, "mu": _params64(mode, prm, nx, nz)["mu"].reshape(-1)}
    if kind == "plugin":
        _, _, norm, g = _exact_gradient(case, prm, src, rec, data, ("mu",), dt)
        return {"gradient": _smooth64(g["mu"]), "misfit": norm, "mu": _params64(mode, prm, nx, nz)["mu"].reshape(-1)}
    if kind == "autograd":
        names = ("mu", "rho") if mode == "sh" else ("lam", "mu", "rho")
        tr, loss, _, g = _exact_gradient(case, prm, src, rec, data, names, 1.0)
        return {"traces": torch.stack(tr), "loss": loss, "gradients": [g[n] for n in names]}
    names = {"sh": ("mu",), "psv": ("lam", "mu"), "spin": ("lam", "mu", "buo", "nu", "mnc", "buo_j")}[mode]
    tr, _, norm, g = _exact_gradient(case, prm, src, rec, data, names, 1.0)
    return {"traces": tr, "misfit": norm, "gradients": [_smooth64(g[n]) for n in names]}
