"""The warp-collective FP64 push at the sizes and operands where its work split
changes: populations around the lane caps and the blocks per SM, powers, roots,
quotients and comparisons on special operands.  The strict push equals the
oracle bit for bit whatever the split, so every comparison is exact."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FRAME, SEED = 7, 20260
FIELDS = ("x", "y", "p", "t", "dt", "mu", "status")


def _population(rng, n, params, special):
    start = {k: np.zeros(n) for k in ("x", "y", "p", "t", "dt", "w", "mu")}
    start["x"] = rng.uniform(0.0, 2.0, n)
    start["y"] = rng.uniform(-2.0, 2.0, n)
    start["p"] = params["p0"] * np.exp(rng.uniform(-0.5, 1.0, n))
    start["t"] = params["mhd_dt"] * (FRAME + rng.uniform(0.0, 0.5, n))
    start["mu"] = rng.uniform(-1.2, 1.2, n)
    start["w"][:] = 1.0
    start["status"] = np.zeros(n, dtype=np.int32)
    start["level"] = np.zeros(n, dtype=np.int32)
    if special and n >= 16:
        start["x"][:4] = (0.0, -0.0, 2.0, -6.5)      # bounds, a signed zero, far outside
        start["y"][:4] = (-2.0, 2.0, 9.0, 1.9999999)
        start["mu"][4:8] = (0.0, -0.0, 0.99, -0.99)
        start["p"][8:12] = (params["p0"], 2.0 * params["p0"], np.nan, -1.0)
        start["status"][12:14] = (1, 2)
        start["t"][14:16] = params["mhd_dt"] * np.array([FRAME + 1.0, FRAME - 0.25])
    return start


def _check(ctx, kpt, oracle, binding, n, focused, closure, stretched, special=False, steps=4,
           **overrides):
    rng = np.random.default_rng(n + 10 * focused + closure)
    params = binding.default_params(kperp_over_kpara=0.05, focused=int(focused), closure=closure)
    if steps:
        params["dt_min_rel"] = params["dt_max_rel"] = (1.0 + 1e-6) / steps
    params.update(overrides)
    ye = kpt.fields.stretched_edges(40, -2.0, 2.0) if stretched else None
    frames = [kpt.fields.harris_field(24, 40, x_range=(0.0, 2.0), y_edges=ye, noise=0.02, seed=s)
              for s in (3, 4)]
    start = _population(rng, n, params, special)
    want = {k: v.copy() for k, v in start.items()}
    grid = oracle.grid(frames[0].x_edges, frames[0].y_edges)
    oracle.push(grid, oracle.table(frames[0], focused), oracle.table(frames[1], focused), params,
                FRAME * params["mhd_dt"], FRAME, SEED, n, want)
    kind = kpt.TABLE_FOCUSED21 if focused else kpt.TABLE_PARKER16
    tables = [ctx.field(f, kind) for f in frames]
    parts = ctx.particles(n)
    settings = kpt.settings_from_dict(params)
    for schedule, blocks in ((kpt.SCHEDULE_REFILL, 0), (kpt.SCHEDULE_REFILL, 1),
                             (kpt.SCHEDULE_SIMPLE, 0)):
        parts.upload(start, n)
        ctx.set_push_schedule(schedule, blocks)
        try:
            stats = ctx.push_interval(parts, tables[0], tables[1], settings, FRAME, SEED)
        finally:
            ctx.set_push_schedule(kpt.SCHEDULE_REFILL, 0)
        got = parts.download()
        for key in FIELDS:
            if key == "mu" and not focused:
                continue
            assert np.array_equal(got[key], want[key], equal_nan=key != "status"), \
                (key, schedule, blocks)
        assert stats.pushed == int(np.sum(start["status"] == 0))
        assert stats.failed == int(np.sum((start["status"] == 0) & (want["status"] != 0)))


# one lane a warp, a few, the step from one block per SM to more, a full wave
@pytest.mark.parametrize("n", [1, 33, 608, 609, 4865, 19457, 40001])
@pytest.mark.parametrize("focused", [False, True])
def test_population_sizes(ctx, kpt, oracle, binding, n, focused):
    _check(ctx, kpt, oracle, binding, n, focused, 0, stretched=n % 2 == 1)


@pytest.mark.parametrize("focused,closure", [(False, 0), (True, 0), (True, 1)])
@pytest.mark.parametrize("overrides", [
    {}, {"time_interpolation": 0}, {"magnetic_dependency": 0}, {"momentum_dependency": 0},
    {"kperp_over_kpara": 0.0}, {"kperp_over_kpara": 1.5}, {"gamma_turb": 2.0},
    {"mhd_dt": 0.3, "p0": 0.37, "charge": 2.0}, {"max_steps": 3}])
def test_special_operands(ctx, kpt, oracle, binding, focused, closure, overrides):
    for stretched in (False, True):
        _check(ctx, kpt, oracle, binding, 300, focused, closure, stretched, special=True,
               **overrides)


@pytest.mark.parametrize("focused,closure", [(False, 0), (True, 0), (True, 1)])
def test_adaptive_steps(ctx, kpt, oracle, binding, focused, closure):
    _check(ctx, kpt, oracle, binding, 130, focused, closure, stretched=True, special=True, steps=0,
           max_steps=60)
