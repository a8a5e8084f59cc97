"""The work that users of this framework have it do, as cases that can be timed.

Families:

* ``push``     one particle store pushed over one or more MHD intervals
               (``Context.push_interval``): Parker or focused transport, FP64
               (strict or contracted arithmetic) or mixed precision, the driver's
               closure, slab QLT or the learned closure;
* ``frame``    one frame of the driver's loop: tables from host fields, injection,
               cell sort, push, split, histogram, summary;
* ``batch``    many independent runs advanced by one launch per interval;
* ``library``  the header library's solvers: a sequence of stochastic steps of a
               ``ParticleSystem`` and its download;
* ``train``    training of the learned closure.

Particles live in torch tensors that the store wraps, so a pass that starts from
a kept state is a device copy away, as in a program that restarts its runs.
``exact`` restates the pushes and the library steps in FP64 torch operations.
"""
from __future__ import annotations

import functools
import importlib
import math

import numpy as np
import torch

kpt = importlib.import_module("kokkos-particletransport_gb300")

DEVICE = "cuda" if torch.cuda.is_available() else "cpu"
FRAME = 100          # first frame of a push
DOUBLES = ("x", "y", "p", "t", "dt", "w", "mu")
INTS = ("status", "level")


# ------------------------------------------------------------------- the cases
def _push(name, **kw):
    case = {"name": name, "family": "push", "focused": False, "precision": "f64",
            "arithmetic": "strict", "closure": "driver", "hidden": 0, "fp16": False,
            "particles": 1 << 16, "nx": 256, "ny": 512, "stretched": True, "substeps": 0,
            "expected_steps": 800, "intervals": 1, "sort": 8, "time_interpolation": True}
    case.update(kw)
    if case["substeps"]:
        case["expected_steps"] = case["substeps"]
    return case


def listed():
    return [
        # a first trial run: a few particles on a small grid, where a call is all latency
        _push("parker_f64_trial", particles=256, nx=32, ny=64, stretched=False, sort=0),
        # the driver's defaults (FP64, Parker, adaptive step) on a uniform square field with
        # a freshly injected population
        _push("parker_f64_driver", particles=1 << 17, nx=1024, ny=1024, stretched=False),
        # focused transport with the driver's own closure in the default arithmetic
        _push("focused_f64_driver", focused=True, particles=60000, nx=250, ny=500,
              stretched=False, substeps=200),
        # the FP64 baseline of the accuracy comparisons: slab QLT, contracted arithmetic
        _push("focused_f64_contracted_qlt", focused=True, closure="qlt", arithmetic="contracted",
              particles=1 << 17, nx=512, ny=1024, substeps=200),
        # production Parker run in mixed precision, adaptive step
        _push("parker_mixed", precision="mixed", particles=1 << 20, nx=1024, ny=2048),
        # focused transport in mixed precision, plain slab-QLT closure, two consecutive
        # intervals of a frame sequence, an uneven particle count
        _push("focused_mixed_qlt", focused=True, closure="qlt", precision="mixed",
              particles=777777, nx=512, ny=1024, substeps=100, intervals=2),
        # the headline configuration: the learned closure at full population
        _push("focused_mixed_learned", focused=True, closure="learned", hidden=32,
              precision="mixed", particles=1 << 22, nx=1024, ny=2048, substeps=100,
              intervals=2),
        # one frame of the driver's loop on a growing population, host fields included
        {"name": "frame_parker_mixed", "family": "frame", "precision": "mixed", "nx": 512,
         "ny": 1024, "stretched": True, "population": 100000, "injected": 25600,
         "expected_steps": 1200},
        # a parameter study: sixteen runs of different sizes in one batch
        {"name": "batch_parker_16", "family": "batch", "runs": 16, "focused": False,
         "smallest": 10000, "largest": 200000, "substeps": 50},
        # the header library's solvers between two diagnostics
        {"name": "library_parker_f64", "family": "library", "solver": "parker",
         "precision": "f64", "particles": 300000, "nx": 512, "ny": 1024, "steps": 40,
         "constant_ratio": False},
        {"name": "library_focus_mixed", "family": "library", "solver": "focus",
         "precision": "mixed", "particles": 400000, "nx": 1024, "ny": 2048, "steps": 250,
         "constant_ratio": False},
        # training the closure at its default width and batch
        {"name": "train_closure", "family": "train", "hidden": 64, "fp16": False,
         "samples": 200000, "steps": 2000, "batch": 8192},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choices(("push", "frame", "batch", "library", "train"), (10, 2, 1, 4, 2))[0]
    nx, ny = _log(rng, 24, 1024), _log(rng, 24, 2048)
    if family == "push":
        focused = rng.random() < 0.6
        precision = rng.choice(("f64", "mixed"))
        closure, hidden = "driver", 0
        if focused:
            closure = rng.choice(("driver", "qlt", "learned"))
            hidden = rng.choice((32, 64)) if closure == "learned" else 0
        most = 150000 if precision == "f64" else 2000000
        particles = _log(rng, 100, most)
        adaptive = not focused and rng.random() < 0.4 and particles < most // 2
        # the step count spread over its range, within the largest case's work
        budget = 2.5e7 if precision == "f64" else 2.5e8
        substeps = 0 if adaptive else max(2, min(_log(rng, 10, 500), int(budget / particles)))
        case = _push("", focused=focused, precision=precision, closure=closure, hidden=hidden,
                     fp16=hidden > 0 and rng.random() < 0.3,
                     arithmetic=rng.choice(("strict", "contracted")), particles=particles,
                     nx=nx, ny=ny, stretched=rng.random() < 0.5, substeps=substeps,
                     intervals=rng.choice((1, 1, 2)), sort=rng.choice((0, 8, 8, 16)),
                     time_interpolation=rng.random() < 0.8)
        del case["name"]
        return case
    if family == "frame":
        return {"family": "frame", "precision": rng.choice(("f64", "mixed")),
                "nx": nx, "ny": ny, "stretched": rng.random() < 0.5,
                "population": _log(rng, 1000, 100000), "injected": _log(rng, 500, 30000),
                "expected_steps": 1200}
    if family == "batch":
        return {"family": "batch", "runs": rng.randint(2, 24),
                "focused": rng.random() < 0.5, "smallest": _log(rng, 500, 10000),
                "largest": _log(rng, 20000, 200000), "substeps": rng.randint(10, 60)}
    if family == "library":
        return {"family": "library", "solver": rng.choice(("parker", "focus")),
                "precision": rng.choice(("f64", "mixed")), "particles": _log(rng, 500, 500000),
                "nx": nx, "ny": ny, "steps": _log(rng, 3, 60),
                "constant_ratio": rng.random() < 0.3}
    return {"family": "train", "hidden": rng.choice((32, 64)),
            "fp16": rng.random() < 0.3, "samples": _log(rng, 5000, 300000),
            "steps": _log(rng, 50, 1500), "batch": _log(rng, 200, 10000)}


# ------------------------------------------------------------------ the inputs
def _edges(n, lower, upper, stretched):
    if not stretched:
        return np.linspace(lower, upper, n + 1)
    # spacing proportional to 1 + 4 y^2 / h^2, finest at the current sheet
    half = 0.5 * (upper - lower)
    s = np.linspace(-1.0, 1.0, n + 1) * math.atan(2.0)
    e = 0.5 * (lower + upper) + half * 0.5 * np.tan(s)
    e[0], e[-1] = lower, upper
    return e


@functools.lru_cache(maxsize=8)
def _sheet(nx, ny, stretched, width=0.1, islands=0.1):
    """A Harris sheet with a guide field, inflow and magnetic islands: cell-centred
    B and V, (6, ny, nx)."""
    xe, ye = _edges(nx, -1.0, 1.0, False), _edges(ny, -2.0, 2.0, stretched)
    x = (0.5 * (xe[1:] + xe[:-1]))[None, :]
    y = (0.5 * (ye[1:] + ye[:-1]))[:, None]
    t, k = np.tanh(y / width), 4.0 * np.pi
    g = islands * np.exp(-y * y / 0.04)
    out = np.zeros((6, ny, nx))
    out[0] = t + np.cos(k * x) * g * (-50.0 * y)
    out[1] = 0.05 * np.sin(np.pi * x) * np.cos(np.pi * y / 4.0) + k * np.sin(k * x) * g
    out[2] = 0.1
    out[3] = 0.1 * x * (1.0 - t * t)
    out[4] = -0.05 * t
    return xe, ye, out


def _frame(nx, ny, stretched, seed, **shape):
    """One frame of a field sequence: the sheet with 1 % noise on every cell."""
    xe, ye, base = _sheet(nx, ny, stretched, **shape)
    noise = np.random.Generator(np.random.SFC64(seed)).standard_normal(base.shape, np.float32)
    cells = base * (1.0 + 0.01 * noise)
    return kpt.fields.CompactField(xe, ye, cells[:3], cells[3:])


def _frames(case, seed):
    return [_frame(case["nx"], case["ny"], case["stretched"], 1000 * seed + k)
            for k in range(case["intervals"] + 1)]


def _settings(case):
    s = kpt.default_settings(kperp_over_kpara=0.05, split_ratio=1.2)
    s.focused = int(case["focused"])
    s.time_interpolation = int(case.get("time_interpolation", True))
    s.closure = {"driver": kpt.CLOSURE_DRIVER, "qlt": kpt.CLOSURE_QLT,
                 "learned": kpt.CLOSURE_SURROGATE}[case.get("closure", "driver")]
    if case["substeps"]:
        # every particle takes exactly this many steps, the last cut to the interval's end
        s.dt_min_rel = s.dt_max_rel = (1.0 + 1e-6) / case["substeps"]
    return s


def _population(n, s, seed, fresh, first_frame=FRAME):
    """n particles spread over the box: at the interval's start, or injected at times
    spread over it (fresh)."""
    rng = np.random.Generator(np.random.SFC64(seed))
    d = np.zeros((len(DOUBLES), n))
    d[0] = rng.uniform(-1.0, 1.0, n)
    d[1] = rng.uniform(-2.0, 2.0, n)
    d[2] = s.p0 * np.exp(rng.uniform(-0.3, 0.7, n))
    d[3] = first_frame * s.mhd_dt + (rng.uniform(0.0, s.mhd_dt, n) if fresh else 0.0)
    d[4] = s.dt_min_rel * s.mhd_dt
    d[5] = 1.0
    d[6] = rng.uniform(-s.mu_max, s.mu_max, n)
    return d


class _State:
    """What a program holds between calls; frees the device objects with itself."""

    def __init__(self, case):
        self.case = case
        self.ctx = kpt.Context(0)
        self.stream = torch.cuda.Stream()
        self.ctx.set_stream(self.stream.cuda_stream)

    def __del__(self):
        try:
            torch.cuda.synchronize()
            self.ctx.close()
        except Exception:
            pass


class _Store:
    """Device arrays of a particle store and the state that every pass starts from."""

    def __init__(self, capacity, population):
        n = population.shape[1]
        self.start = torch.from_numpy(population).to(DEVICE)
        self.doubles = torch.zeros((len(DOUBLES), capacity), dtype=torch.float64, device=DEVICE)
        self.ints = torch.full((2, capacity), 2, dtype=torch.int32, device=DEVICE)
        self.ints[1] = 0
        self.start_ints = self.ints.clone()
        self.start_ints[0, :n] = 0
        self.n = n

    def restore(self):
        self.doubles[:, :self.n].copy_(self.start)
        self.ints.copy_(self.start_ints)

    def wrap(self, ctx, lo=0, hi=None):
        hi = self.doubles.shape[1] if hi is None else hi
        ptrs = {k: self.doubles[i, lo:].data_ptr() for i, k in enumerate(DOUBLES)}
        ptrs |= {k: self.ints[i, lo:].data_ptr() for i, k in enumerate(INTS)}
        names = dict(zip(DOUBLES + INTS, ("x", "y", "p", "t", "step_dt", "weight", "mu",
                                          "status", "split_level")))
        return ctx.wrap_particles(hi - lo, hi - lo, {names[k]: v for k, v in ptrs.items()})

    def outputs(self):
        return {k: self.doubles[i] for i, k in enumerate(DOUBLES)} | \
               {k: self.ints[i] for i, k in enumerate(INTS)}


def prepare(case, seed):
    return globals()["_prepare_" + case["family"]](case, int(seed))


def run(state):
    with torch.cuda.stream(state.stream):
        return globals()["_run_" + state.case["family"]](state)


# ---------------------------------------------------------------------- push
def _prepare_push(case, seed):
    st = _State(case)
    ctx = st.ctx
    st.settings = s = _settings(case)
    if case["arithmetic"] == "contracted":
        ctx.set_fp64_arithmetic(kpt.FP64_CONTRACTED)
    if case["closure"] == "learned":
        st.network = ctx.train_surrogate(
            s, samples=100000, steps=1000, batch=4096, hidden_width=case["hidden"],
            element_type=kpt.SURROGATE_FP16 if case["fp16"] else kpt.SURROGATE_BF16,
            mu_cut=0.005, b_lo=0.005)
        ctx.set_surrogate(st.network)
    kind = kpt.TABLE_FOCUSED21 if case["focused"] else kpt.TABLE_PARKER16
    prec = kpt.PRECISION_MIXED if case["precision"] == "mixed" else kpt.PRECISION_F64
    st.tables = [ctx.field(f, kind, prec) for f in _frames(case, seed)]
    st.store = _Store(case["particles"],
                      _population(case["particles"], s, seed, fresh=not case["substeps"]))
    st.parts = st.store.wrap(ctx)
    st.seed = seed
    torch.cuda.synchronize()
    return st


def _run_push(st):
    case, ctx = st.case, st.ctx
    st.store.restore()
    out = {}
    for k in range(case["intervals"]):
        lower, upper = st.tables[k], st.tables[k + 1]
        if case["sort"]:
            ctx.sort(st.parts, lower, case["sort"], case["sort"])
        stats = ctx.push_interval(st.parts, lower, upper, st.settings, FRAME + k, st.seed)
        out[f"steps{k}"] = int(stats.particle_steps)
        out[f"longest{k}"] = int(stats.max_steps)
        out[f"failed{k}"] = int(stats.failed)
    if case["closure"] == "learned":
        judge = ctx.surrogate_judge()
        out |= {k: judge[k] for k in ("evaluations", "judged", "fallbacks")}
    return out | st.store.outputs()


# --------------------------------------------------------------------- frame
def _prepare_frame(case, seed):
    st = _State(case)
    st.fields = [_frame(case["nx"], case["ny"], case["stretched"], 1000 * seed + k)
                 for k in range(2)]
    st.settings = s = kpt.default_settings(kperp_over_kpara=0.05, split_ratio=1.2)
    st.prec = kpt.PRECISION_MIXED if case["precision"] == "mixed" else kpt.PRECISION_F64
    st.lower = st.ctx.field(st.fields[0], kpt.TABLE_PARKER16, st.prec)
    n = case["population"]
    st.store = _Store(2 * n + case["injected"], _population(n, s, seed, fresh=False))
    st.parts = st.store.wrap(st.ctx)
    st.seed = seed
    torch.cuda.synchronize()
    return st


def _run_frame(st):
    # the frame's upper field arrives from the host, as the driver reads one per frame
    case, ctx, s = st.case, st.ctx, st.settings
    st.store.doubles.zero_()
    st.store.restore()
    st.parts.set_count(case["population"])
    upper = ctx.field(st.fields[1], kpt.TABLE_PARKER16, st.prec)
    injected = ctx.inject(st.parts, st.lower, s, case["injected"], FRAME, st.seed)
    ctx.sort(st.parts, st.lower, 8, 8)
    stats = ctx.push_interval(st.parts, st.lower, upper, s, FRAME, st.seed)
    split, skipped = ctx.split(st.parts, s)
    bins = ctx.histogram(st.parts, s.pmin, s.pmax, 128)
    summary = ctx.summarize(st.parts)
    upper.close()
    return {"injected": injected, "steps": int(stats.particle_steps),
            "longest": int(stats.max_steps), "failed": int(stats.failed), "split": split,
            "skipped": skipped, "count": st.parts.count, "bins": bins,
            "summary": summary} | st.store.outputs()


# --------------------------------------------------------------------- batch
def _batch_runs(case, seed):
    # the study's sizes are the case's; the seed gives fields, populations and noise
    rng = np.random.default_rng(case["runs"])
    sizes = ((128, 128), (256, 512), (512, 1024))
    runs = []
    for r in range(case["runs"]):
        nx, ny = sizes[int(rng.integers(len(sizes)))]
        n = int(round(math.exp(rng.uniform(math.log(case["smallest"]),
                                           math.log(case["largest"])))))
        runs.append((nx, ny, n, float(rng.choice((0.06, 0.1, 0.16))), 1000 * seed + r))
    return runs


def _batch_settings(case):
    return _settings({"focused": case["focused"], "substeps": case["substeps"],
                      "closure": "qlt" if case["focused"] else "driver"})


def _prepare_batch(case, seed):
    st = _State(case)
    ctx, s = st.ctx, _batch_settings(case)
    kind = kpt.TABLE_FOCUSED21 if case["focused"] else kpt.TABLE_PARKER16
    runs = _batch_runs(case, seed)
    # each run's slice starts on a 32-particle boundary of the shared arrays
    ends = np.cumsum([(n + 31) // 32 * 32 for _, _, n, _, _ in runs])
    st.frame = FRAME
    st.store = _Store(int(ends[-1]), np.zeros((len(DOUBLES), int(ends[-1]))))
    st.batch = ctx.batch()
    st.keep = []
    for (nx, ny, n, width, key), end in zip(runs, ends):
        lo = int(end) - (n + 31) // 32 * 32
        st.store.doubles[:, lo:lo + n].copy_(torch.from_numpy(_population(n, s, key, False)))
        st.store.ints[0, lo:lo + n] = 0
        parts = st.store.wrap(ctx, lo, lo + n)
        table = ctx.field(_frame(nx, ny, False, key, width=width), kind, kpt.PRECISION_MIXED)
        st.batch.add_run(parts, table, table, s, key, FRAME)
        st.keep.append((parts, table))
    torch.cuda.synchronize()
    return st


def _run_batch(st):
    # the runs go on from where the last pass left them, one interval further
    st.batch.run(1)
    return {"frame": st.batch.frame(0)} | st.store.outputs()


# ------------------------------------------------------------------- library
def _library_basis(case, seed):
    """Smooth periodic coefficient fields in the solvers' packed order, with seeded
    amplitudes: (points, 18 or 27) over the ghosted cells."""
    nx, ny = case["nx"], case["ny"]
    rng = np.random.default_rng(seed)
    a = rng.uniform(0.8, 1.2, 4)
    x = (-1.0 + (np.arange(-2, nx + 2) + 0.5) * 2.0 / nx)[None, :]
    y = (-2.0 + (np.arange(-2, ny + 2) + 0.5) * 4.0 / ny)[:, None]
    kx, ky = np.pi, np.pi / 2.0
    sx, cx, sy, cy = np.sin(kx * x), np.cos(kx * x), np.sin(ky * y), np.cos(ky * y)
    b = np.zeros((ny + 4, nx + 4, 3))
    b[..., 0] = np.tanh(sy / 0.3) + 0.05
    b[..., 1] = 0.1 * a[0] * sx * cy
    b[..., 2] = 0.2
    kpar = 0.01 * a[1] * (1.2 + sx * cy)
    divv = 0.1 * a[2] * cx * sy
    if case["solver"] == "parker":
        out = np.zeros((ny + 4, nx + 4, 18))
        out[..., 0:3] = b
        out[..., 3] = 0.1 * cx
        out[..., 4] = -0.05 * sy
        out[..., 6] = 0.02 * sx * cy
        out[..., 7] = 0.02 * cx * sy
        out[..., 8] = 0.01 * sy
        out[..., 9] = 1e-3 * a[3] * cx
        out[..., 10] = 1e-3 * sy
        if not case["constant_ratio"]:
            out[..., 12] = 5e-4 * sx
            out[..., 13] = 5e-4 * cy
        out[..., 15] = kpar
        out[..., 16] = 0.05 * kpar if case["constant_ratio"] else 1e-3 * (1.1 + cx)
        out[..., 17] = divv
        return out.reshape(-1, 18)
    out = np.zeros((ny + 4, nx + 4, 27))
    mag = np.sqrt((b * b).sum(-1))
    out[..., 0:3] = b
    out[..., 3:6] = b / mag[..., None]
    out[..., 6] = 0.1 * cx
    out[..., 7] = -0.05 * sy
    out[..., 9] = 0.01 * sx
    out[..., 10] = 0.01 * a[3] * cy
    out[..., 12] = 0.005 * cx * cy
    out[..., 13] = 0.005 * sx
    out[..., 14] = 0.002
    out[..., 15] = 1e-4 * sy
    out[..., 16] = 1e-4 * cx
    out[..., 18] = mag
    out[..., 19] = kpar
    out[..., 20] = 5e-4 * (1.1 + cx)
    out[..., 21] = divv
    out[..., 22] = 0.2 * sx * cy
    out[..., 23] = 0.05 * cy
    out[..., 24] = 0.02 * sx
    out[..., 25] = 0.1 * (1.0 + 0.5 * sx * sy)
    out[..., 26] = 0.05 * (1.0 + 0.2 * cx)
    return out.reshape(-1, 27)


def _library_state(case, seed):
    n = case["particles"]
    rng = np.random.default_rng(seed)
    state = {"id": np.arange(n, dtype=np.uint64)}
    state |= {k: np.zeros(n) for k in kpt.SYSTEM_DOUBLE_FIELDS}
    state |= {k: np.zeros(n, dtype=np.int32) for k in kpt.SYSTEM_INT_FIELDS}
    state["x"] = rng.uniform(-1.0, 1.0, n)
    state["y"] = rng.uniform(-2.0, 2.0, n)
    for k in ("prev", "prevstep"):
        state[k + "_x"], state[k + "_y"] = state["x"].copy(), state["y"].copy()
    state["p"] = np.exp(rng.uniform(math.log(0.05), math.log(3.0), n))
    state["mu"] = rng.uniform(-1.0, 1.0, n)
    state["w"] = np.ones(n)
    return state


def _prepare_library(case, seed):
    st = _State(case)
    ctx, n = st.ctx, case["particles"]
    st.grid = ctx.grid(np.linspace(-1.0, 1.0, case["nx"] + 1),
                       np.linspace(-2.0, 2.0, case["ny"] + 1), (1, 1))
    make = ctx.parker_solver if case["solver"] == "parker" else ctx.focus_solver
    st.solver = make(st.grid, _library_basis(case, seed), case["constant_ratio"])
    if case["precision"] == "mixed":
        st.solver.set_precision(kpt.PRECISION_MIXED)
    st.system = ctx.system(n, n)
    st.system.upload(_library_state(case, seed))
    st.step, st.seed = 0, seed
    torch.cuda.synchronize()
    return st


def _run_library(st):
    # the system goes on from where the last pass left it
    dts = st.solver.advance_stochastic_steps(st.system, st.seed, st.step, st.case["steps"])
    st.step += st.case["steps"]
    out = st.system.download()
    out["id"] = out["id"].view(np.int64)
    return out | {"dts": dts}


# --------------------------------------------------------------------- train
def _prepare_train(case, seed):
    st = _State(case)
    st.settings = kpt.default_settings(kperp_over_kpara=0.05, focused=1,
                                       closure=kpt.CLOSURE_SURROGATE)
    st.seed = seed
    return st


def _run_train(st):
    case = st.case
    net = st.ctx.train_surrogate(
        st.settings, samples=case["samples"], steps=case["steps"], batch=case["batch"],
        hidden_width=case["hidden"], seed=st.seed,
        element_type=kpt.SURROGATE_FP16 if case["fp16"] else kpt.SURROGATE_BF16)
    params, norm = net.parameters()
    out = {"parameters": params, "offset": norm["out_offset"].astype(np.float32),
           "scale": norm["out_scale"].astype(np.float32)}
    net.close()
    return out


# ---------------------------------------------------------------------- work
def work(case):
    """State and tables read and written once; the arithmetic of every substep once."""
    family = case["family"]
    if family in ("push", "frame"):
        focused = case.get("focused", False)
        comps = 21 if focused else 16
        elem = 4 if case["precision"] == "mixed" else 8
        points = (case["nx"] + 4) * (case["ny"] + 4)
        intervals = case.get("intervals", 1)
        n = case["particles"] if family == "push" else case["population"] + case["injected"]
        flop = 2 * 2 * 4 * comps + (450 if focused else 250)
        if case.get("closure") == "learned":
            h = case["hidden"]
            flop += 2 * (5 * h + h * h + 3 * h)
        data = intervals * (n * 120 + 2 * points * comps * elem)
        if family == "frame":
            data += 48 * case["nx"] * case["ny"]
        mean = case["expected_steps"] * (1.0 if case.get("substeps") else 0.5)
        return {"bytes": data, "flops": n * intervals * mean * flop}
    if family == "batch":
        n = case["runs"] * (case["largest"] - case["smallest"]) / \
            math.log(case["largest"] / case["smallest"])
        comps = 21 if case["focused"] else 16
        points = case["runs"] * 0.25e6
        return {"bytes": n * 120 + points * comps * 4,
                "flops": n * case["substeps"] * (16 * comps + (450 if case["focused"] else 250))}
    if family == "library":
        comps = 18 if case["solver"] == "parker" else 27
        elem = 4 if case["precision"] == "mixed" else 8
        points = (case["nx"] + 4) * (case["ny"] + 4)
        # every step reads and writes positions, their histories, momentum and cosine
        per = 2 * 8 * (7 if case["solver"] == "parker" else 8) + 4
        return {"bytes": case["steps"] * (case["particles"] * per +
                                          min(points, 4 * case["particles"]) * comps * elem),
                "flops": case["steps"] * case["particles"] *
                (8 * comps + (200 if case["solver"] == "parker" else 500))}
    h = case["hidden"]
    per = 2 * (5 * h + h * h + 3 * h)
    return {"bytes": case["steps"] * case["batch"] * 32.0 + case["samples"] * 32.0,
            "flops": 3.0 * per * case["batch"] * case["steps"]}


# --------------------------------------------------------------------- exact
def exact(case, seed):
    """The outputs in FP64 torch operations; None where they take too long that way
    (tens of thousands of substeps one after another), follow from the library's own
    trained network, or where an FP32 run has no FP64 twin: pitch angles near mu = 0, where
    dD/dmu is singular, amplify the rounding of a step by orders of magnitude within some
    tens of steps (and set the lockstep solver's dt)."""
    seed = int(seed)
    if case["family"] == "push":
        steps = case["substeps"] or 4000
        if case["focused"] and case["precision"] == "mixed" and case["intervals"] * steps > 50:
            return None
        if case["closure"] == "learned" or \
                case["intervals"] * steps * max(1.0, case["particles"] / 4e5) > 6000:
            return None
        s = _settings(case)
        d = _population(case["particles"], s, seed, fresh=not case["substeps"])
        frames = _frames(case, seed)
        state = {k: torch.from_numpy(d[i].copy()).to(DEVICE) for i, k in enumerate(DOUBLES)}
        for k in range(case["intervals"]):
            _exact_push(state, frames[k], frames[k + 1], s, FRAME + k, seed)
        return state
    if case["family"] == "batch":
        s = _batch_settings(case)
        runs = _batch_runs(case, seed)
        if case["focused"] or sum(case["substeps"] * max(1.0, r[2] / 4e5) for r in runs) > 2000:
            return None
        parts = []
        for nx, ny, n, width, key in runs:
            d = _population(n, s, key, False)
            state = {k: torch.from_numpy(d[i].copy()).to(DEVICE) for i, k in enumerate(DOUBLES)}
            field = _frame(nx, ny, False, key, width=width)
            _exact_push(state, field, field, s, FRAME, key)
            pad = (-n) % 32
            parts.append({k: torch.nn.functional.pad(v, (0, pad)) for k, v in state.items()})
        return {k: torch.cat([p[k] for p in parts]) for k in DOUBLES}
    if case["family"] == "library":
        if case["steps"] * max(1.0, case["particles"] / 4e5) > 3000:
            return None
        if case["solver"] == "focus" and case["precision"] == "mixed" and case["steps"] > 5:
            return None
        return _exact_library(case, seed)
    return None


def _philox(block, index, frame, tag, seed):
    """Philox4x32-10 words in int64 tensors: counter (block, index, frame, tag)."""
    mask = 0xFFFFFFFF
    c = [block, index, torch.full_like(index, frame), torch.full_like(index, tag)]
    k0, k1 = seed & mask, (seed >> 32) & mask
    for _ in range(10):
        p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
        c = [((p1 >> 32) & mask) ^ c[1] ^ k0, p1 & mask,
             ((p0 >> 32) & mask) ^ c[3] ^ k1, p0 & mask]
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    return c


def _u01(lo, hi):
    return (((hi << 21) | (lo >> 11)).double()) * 2.0 ** -53


def _exact_axis(edges):
    """(lower, width, n, ghosted centres or None for a uniform axis)."""
    n, w = edges.size - 1, edges[-1] - edges[0]
    steps = np.diff(edges)
    if np.max(np.abs(steps - w / n)) < 1e-12:
        return float(edges[0]), float(w), n, None
    faces = np.concatenate([edges[n - 2:n] - w, edges, edges[1:3] + w])
    return float(edges[0]), float(w), n, torch.from_numpy(0.5 * (faces[1:] + faces[:-1])).to(DEVICE)


def _exact_table(field, focused):
    """Cell-centred coefficients and their centred differences, (ny, nx, components)."""
    b = [torch.from_numpy(np.ascontiguousarray(c)).to(DEVICE) for c in field.b]
    v = [torch.from_numpy(np.ascontiguousarray(c)).to(DEVICE) for c in field.v]
    mag = torch.sqrt(b[0] * b[0] + b[1] * b[1] + b[2] * b[2])
    spans = []
    for edges in (field.x_edges, field.y_edges):
        lower, w, n, centres = _exact_axis(edges)
        spans.append(2.0 * w / n if centres is None else centres[3:n + 3] - centres[1:n + 1])

    def dx(f):
        return (torch.roll(f, -1, 1) - torch.roll(f, 1, 1)) / spans[0]

    def dy(f):
        span = spans[1]
        return (torch.roll(f, -1, 0) - torch.roll(f, 1, 0)) / \
            (span if isinstance(span, float) else span[:, None])
    if focused:
        comps = v + b + [mag]
        for f in (v[0], v[1], v[2], b[0], b[1], b[2], mag):
            comps += [dx(f), dy(f)]
    else:
        comps = [v[0], v[1], b[0], b[1], b[2], mag, dx(v[0]), dy(v[1])]
        for f in (b[0], b[1], b[2], mag):
            comps += [dx(f), dy(f)]
    return torch.stack(comps, -1)


def _exact_cell(axis, pos):
    lower, w, n, centres = axis
    q = pos + 0.5 * w / n
    q = torch.where(q >= lower + w, q - w, q)
    if centres is None:
        logical = (q - lower) / (w / n) - 0.5
        lo = torch.floor(logical)
        return lo.long(), logical - lo
    k = torch.searchsorted(centres, q.contiguous(), right=True) - 1
    return k - 2, (q - centres[k]) / (centres[k + 1] - centres[k])


def _exact_push(state, field0, field1, s, frame, seed):
    """One interval of the driver's Parker or focused push, in place."""
    focused = s.focused != 0
    ax, ay = _exact_axis(field0.x_edges), _exact_axis(field0.y_edges)
    tables = (_exact_table(field0, focused), _exact_table(field1, focused))
    start = frame * s.mhd_dt
    end = start + s.mhd_dt
    dt_lo, dt_hi = s.dt_min_rel * s.mhd_dt, s.dt_max_rel * s.mhd_dt
    dx, dy = ax[1] / ax[2], ay[1] / ay[2]
    g, sq3 = s.gamma_turb, math.sqrt(3.0)
    index = torch.arange(state["x"].numel(), device=DEVICE)
    if focused:
        state["mu"].clamp_(-s.mu_max, s.mu_max)
    left = index[state["t"] < end]
    step = 0
    while left.numel():
        x, y, p, t, mu = (state[k][left] for k in ("x", "y", "p", "t", "mu"))
        i0, w0 = _exact_cell(ax, x)
        j0, w1 = _exact_cell(ay, y)
        i, j = (i0 % ax[2], (i0 + 1) % ax[2]), (j0 % ay[2], (j0 + 1) % ay[2])
        weights = ((1 - w0) * (1 - w1), w0 * (1 - w1), (1 - w0) * w1, w0 * w1)

        def sample(table):
            corners = (table[j[0], i[0]], table[j[0], i[1]], table[j[1], i[0]], table[j[1], i[1]])
            return sum(wt[:, None] * cv for wt, cv in zip(weights, corners))
        c = sample(tables[0])
        if s.time_interpolation:
            u = ((t - start) / s.mhd_dt).clamp(0.0, 1.0)[:, None]
            c = (1.0 - u) * c + u * sample(tables[1])
        c = c.t().contiguous()
        if focused:
            vx, vy, _, bx, by, bz, b, vxx, vxy, vyx, vyy, vzx, vzy, bxx, bxy, byx, byy, bzx, \
                bzy, bmx, bmy = c
        else:
            vx, vy, bx, by, bz, b, vxx, vyy, bxx, bxy, byx, byy, bzx, bzy, bmx, bmy = c
        ib = 1.0 / b
        ib2, ib3 = ib * ib, ib * ib * ib
        kpara = s.kpara0 * torch.ones_like(p)
        gx, gy = torch.zeros_like(p), torch.zeros_like(p)
        if s.magnetic_dependency == 1:
            kpara = kpara * b ** (g - 2.0)
            gx, gy = bmx * ib * (g - 2.0), bmy * ib * (g - 2.0)
        if s.momentum_dependency == 1:
            kpara = kpara * (p / s.p0) ** (3.0 - g)
        kperp = kpara * s.kperp_over_kpara
        spara, sperp = torch.sqrt(2.0 * kpara), torch.sqrt(2.0 * kperp)
        kd = -kperp if focused else kpara - kperp
        kxx = kperp * gx + kd * gx * bx * bx * ib2 + 2 * kd * bx * (bxx * b - bx * bmx) * ib3
        kyy = kperp * gy + kd * gy * by * by * ib2 + 2 * kd * by * (byy * b - by * bmy) * ib3
        kxyx = kd * gx * bx * by * ib2 + kd * ((bxx * by + bx * byx) * ib2 -
                                               2 * bx * by * bmx * ib3)
        kxyy = kd * gy * bx * by * ib2 + kd * ((bxy * by + bx * byy) * ib2 -
                                               2 * bx * by * bmy * ib3)
        drift = torch.sqrt((s.drift_param1 * s.p0 / p) ** 2 +
                           (s.drift_param2 * s.p0 * s.p0 / (p * p)) ** 2)
        divv = vxx + vyy
        big = torch.full_like(p, math.inf)
        if focused:
            mu2 = mu * mu
            f1, f2 = 0.5 * (1 - mu2), 0.5 * (3 * mu2 - 1)
            cx, cy, cz = bx * bxx + by * bxy, bx * byx + by * byy, bx * bzx + by * bzy
            curl = bx * bzy - by * bzx + bz * (byx - bxy)
            vd = 1.0 / s.charge / drift
            vdx = vd * (f1 * (-bz * bmy) * ib2 + mu2 * (by * cz - bz * cy) * ib3 +
                        f1 * bx * curl * ib3)
            vdy = vd * (f1 * (bz * bmx) * ib2 + mu2 * (bz * cx - bx * cz) * ib3 +
                        f1 * by * curl * ib3)
            speed = s.particle_v0 * p / s.p0
            along = speed * mu * ib
            xr = vx + vdx + along * bx + kxx + kxyy
            yr = vy + vdy + along * by + kxyx + kyy
            bb = (bx * (bx * vxx + by * vxy) + by * (bx * vyx + by * vyy) +
                  bz * (bx * vzx + by * vzy)) * ib2
            bv = (bx * (vx * vxx + vy * vxy) + by * (vx * vyx + vy * vyy) +
                  bz * (vx * vzx + vy * vzy)) * ib
            pr = -p * (f1 * divv + f2 * bb + mu * bv / speed)
            mr = speed * (-(bx * bmx + by * bmy) * ib2) + mu * divv - 3 * mu * bb - 2 * bv / speed
            mr = mr * f1
            am, sign = mu.abs(), torch.sign(mu)
            if s.closure == 1:
                omega = s.qlt_omega0 * b / torch.sqrt(1 + p * p)
                gk, reg = s.qlt_spectral_index, am + s.qlt_h0
                xi = omega * s.qlt_lc / speed
                den = reg ** gk + xi ** gk
                pre = 0.25 * omega * s.qlt_sigma2 * gk * math.sin(math.pi / gk)
                duu = pre * (1 - mu2) * xi * reg ** (gk - 1) / den
                ddu = duu * (-2 * mu / (1 - mu2) +
                             sign * ((gk - 1) / reg - gk * reg ** (gk - 1) / den))
            else:
                e = am ** (g - 1) + 0.2
                duu = s.duu0 * (1 - mu2) * e
                ddu = s.duu0 * (-2 * mu * e + sign * (1 - mu2) * am ** (g - 2))
                ddu = torch.where(mu == 0.0, torch.zeros_like(ddu), ddu)
                norm = torch.ones_like(p)
                if s.magnetic_dependency == 1:
                    norm = norm * b ** (2 - g)
                if s.momentum_dependency == 1:
                    norm = norm * (p / s.p0) ** (g - 1)
                duu, ddu = duu * norm, ddu * norm
            mr = mr + ddu
            scale = torch.where(sperp > 0, sperp, spara)
            dt = torch.minimum((0.5 * dx / scale) ** 2, (0.5 * dy / scale) ** 2)
            for bound in ((scale / xr) ** 2, (scale / yr) ** 2, 0.1 * p / pr.abs(),
                          0.1 / mr.abs(), 2 * duu / mr ** 2):
                dt = torch.minimum(dt, bound)
            fixed = (xr == 0) | (yr == 0) | (pr == 0) | (mr == 0)
        else:
            vd = 1.0 / (3.0 * s.charge) / drift
            vdx = vd * (bzy * ib2 - 2 * bz * bmy * ib3)
            vdy = vd * (-bzx * ib2 + 2 * bz * bmx * ib3)
            xr = vx + vdx + kxx + kxyy
            yr = vy + vdy + kxyx + kyy
            pr = -p * divv / 3.0
            scale = torch.where(sperp > 0, sperp, spara)
            dt = torch.minimum((0.5 * dx / spara) ** 2, (0.5 * dy / spara) ** 2)
            for bound in ((scale / xr) ** 2, (scale / yr) ** 2, 0.1 * p / pr.abs()):
                dt = torch.minimum(dt, bound)
            fixed = (xr == 0) | (yr == 0) | (pr == 0)
        dt = torch.where(fixed, torch.full_like(dt, dt_lo), torch.minimum(dt, big))
        dt = dt.clamp(dt_lo, dt_hi)
        state["dt"][left] = dt
        rest = end - t
        last = dt > rest
        dt = torch.where(last, rest, dt)
        sdt = torch.sqrt(dt)
        block = torch.full_like(left, 2 * step)
        r0 = _philox(block, left, frame, 2, seed)
        r1 = _philox(block + 1, left, frame, 2, seed)
        n1 = -sq3 + 2 * sq3 * _u01(r0[0], r0[1])
        n2 = -sq3 + 2 * sq3 * _u01(r0[2], r0[3])
        if focused:
            n4 = -sq3 + 2 * sq3 * _u01(r1[2], r1[3])
            hx, hy, hz = bx * ib, by * ib, bz * ib
            hxy = torch.sqrt(hx * hx + hy * hy)
            f = torch.where(hxy > 0, sperp / hxy * sdt, torch.zeros_like(p))
            x = x + xr * dt + f * (-hx * hz * n1 - by * n2)
            y = y + yr * dt + f * (-hy * hz * n1 + bx * n2)
            mu = (mu + mr * dt + n4 * torch.sqrt(2 * duu) * sdt).clamp(-s.mu_max, s.mu_max)
            state["mu"][left] = mu
        else:
            n3 = -sq3 + 2 * sq3 * _u01(r1[0], r1[1])
            sd = torch.sqrt(2 * (kpara - kperp))
            x = x + xr * dt + n1 * sperp * sdt + n3 * sd * sdt * bx * ib
            y = y + yr * dt + n2 * sperp * sdt + n3 * sd * sdt * by * ib
        p = (p + pr * dt).clamp(min=0.25 * s.p0)
        state["x"][left] = x - torch.floor((x - ax[0]) / ax[1]) * ax[1]
        state["y"][left] = y - torch.floor((y - ay[0]) / ay[1]) * ay[1]
        state["p"][left] = p
        t = torch.where(last, torch.full_like(t, end), t + dt)
        state["t"][left] = t
        step += 1
        left = left[t < end]


def _exact_library(case, seed):
    """The lockstep solvers on the uniform periodic grid: ParkerSolver or
    FocusTransportSolver, speed of light, mass and charge 1."""
    nx, ny = case["nx"], case["ny"]
    basis = torch.from_numpy(_library_basis(case, seed)).to(DEVICE)
    st = {k: torch.from_numpy(v).to(DEVICE) for k, v in _library_state(case, seed).items()
          if v.dtype == np.float64}
    n = case["particles"]
    index = torch.arange(n, device=DEVICE)
    courant, focus = 0.3, case["solver"] == "focus"
    widths = (2.0 / nx, 4.0 / ny)
    gk, h0 = 5.0 / 3.0, 1e-6
    dts = []

    def wrap():
        for k, lower, w in (("x", -1.0, 2.0), ("y", -2.0, 4.0)):
            shift = -torch.floor((st[k] - lower) / w) * w
            for name in (k, "prev_" + k, "prevstep_" + k):
                st[name] = st[name] + shift

    def reflect(m):
        for _ in range(8):
            m = torch.where(m > 1.0, 2.0 - m, m)
            m = torch.where(m < -1.0, -2.0 - m, m)
        return m
    for step in range(case["steps"]):
        wrap()
        lx, ly = (st["x"] + 1.0) / widths[0] - 0.5, (st["y"] + 2.0) / widths[1] - 0.5
        i, j = torch.floor(lx), torch.floor(ly)
        wx, wy = lx - i, ly - j
        at = (j.long() + 2) * (nx + 4) + i.long() + 2
        c = ((1 - wx) * (1 - wy))[:, None] * basis[at] + (wx * (1 - wy))[:, None] * basis[at + 1] \
            + ((1 - wx) * wy)[:, None] * basis[at + nx + 4] \
            + (wx * wy)[:, None] * basis[at + nx + 5]
        c = c.t().contiguous()
        p = st["p"].abs()
        gamma = torch.sqrt(1 + p * p)
        speed = p / gamma
        third, ninth = gamma ** (1.0 / 3.0), gamma ** (1.0 / 9.0)
        perp = third if case["constant_ratio"] else ninth
        if focus:
            mu = reflect(st["mu"])
            mag = torch.sqrt((c[3:6] ** 2).sum(0))
            d = c[3:6] / mag
            kpar, kperp = c[19] * third, c[20] * perp
            mu2 = mu * mu
            pre = p * speed
            total = speed * mu * d + c[6:9] + pre * (0.5 * (1 - mu2) * c[9:12] +
                                                     mu2 * c[12:15]) + perp * c[15:18]
            keff = [torch.clamp(1 - d[k] * d[k], min=0.0) * kperp for k in range(2)]
            prate = -p * (0.5 * (1 - mu2) * (c[21] - c[23]) + mu2 * c[23] + mu * c[24] / speed)
            omega = c[18] / gamma
            xi = omega * c[26] / speed
            strength = 0.25 * omega * c[25] * gk * math.sin(math.pi / gk)

            def pitch(m):
                m = reflect(m)
                om = 1 - m * m
                focusing = 0.5 * om * (-speed * c[22] + m * c[21] - 3 * m * c[23] -
                                       2 * c[24] / speed)
                reg = m.abs() + h0
                den = reg ** gk + xi ** gk
                D = strength * om * xi * reg ** (gk - 1) / den
                dD = D * (-2 * m / om + torch.sign(m) * ((gk - 1) / reg -
                                                         gk * reg ** (gk - 1) / den))
                dD = torch.where((D != 0) & (m != 0), dD, torch.zeros_like(dD))
                return D, focusing + dD
            D, rate = pitch(mu)
            inf = torch.full_like(p, 1e300)
            bound = torch.minimum(torch.where(prate != 0, p / prate.abs(), inf),
                                  torch.where(rate != 0, 1.0 / rate.abs(), inf))
            bound = torch.minimum(bound, torch.where(D > 0, 0.05 / D, inf))
            bound = torch.minimum(bound, torch.where(D > 0, 20 * D / rate ** 2, inf))
        else:
            b2 = (c[0:3] ** 2).sum(0)
            d = c[0:3] / torch.sqrt(b2)
            kpar, kperp = c[15] * third, c[16] * perp
            diff = third * c[9:12]
            if not case["constant_ratio"]:
                diff = diff + ninth * c[12:15]
            total = c[3:6] + p * speed / 3.0 * c[6:9] + diff
            keff = [kperp + (kpar - kperp) * d[k] * d[k] for k in range(2)]
            prate = -(p / 3.0) * c[17]
            bound = 3.0 / c[17].abs()
        for k in range(2):
            bound = torch.minimum(bound, (0.5 * widths[k]) ** 2 / (2 * keff[k]))
            bound = torch.minimum(bound, widths[k] / total[k].abs())
        dt = courant * float(bound.min())
        dts.append(dt)
        z = []
        for block in range(2):
            r = _philox(torch.full_like(index, block), index, step, 3, seed)
            radius = torch.sqrt(-2 * torch.log(1.0 - _u01(r[0], r[1])))
            angle = 2 * math.pi * _u01(r[2], r[3])
            z += [radius * torch.cos(angle), radius * torch.sin(angle)]
        for k in ("x", "y"):
            st["prevstep_" + k], st["prev_" + k] = st["prev_" + k], st[k]
        along = z[0] * d[0] + z[1] * d[1] + z[2] * d[2]
        sp = torch.sqrt(2 * kperp * dt)
        if focus:
            inc = [sp * (z[k] - along * d[k]) for k in range(2)]
            trial = mu
            for _ in range(3):
                D, rate = pitch(trial)
                trial = reflect(mu + dt * rate + torch.sqrt(2 * D.clamp(min=0) * dt) * z[3])
            st["mu"] = trial
        else:
            rep = torch.sqrt(2 * kpar * dt) * z[3] - sp * along
            inc = [sp * z[k] + rep * d[k] for k in range(2)]
        st["x"] = st["x"] + dt * total[0] + inc[0]
        st["y"] = st["y"] + dt * total[1] + inc[1]
        st["p"] = (p + dt * prate).clamp(min=0.0)
        wrap()
    return {k: st[k] for k in kpt.SYSTEM_DOUBLE_FIELDS} | {"dts": np.array(dts)}
