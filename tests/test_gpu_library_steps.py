"""The library step's two launches over the sizes where their pieces meet.

The terms pass keeps a row of values per term (rows padded to 32 particles),
folds the local dt bounds by block and lets the last block form the step's dt
and clear the words for the next step.  Sizes around a warp, a block and one
pass of the largest grid (152 * 32 blocks of 256):

* the dt of a system is the smaller of its halves' dts, exactly (the minimum
  commutes with the product by the Courant number);
* steps replayed in one call equal steps called one by one, bit for bit, also
  on a solver whose last step failed (no particle left to bound the dt).
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import lib_grid, load_golden

pytestmark = pytest.mark.gpu

SIZES = (1, 31, 33, 256, 257, 152 * 32 * 256 + 33)


def _state(kpt, data, n):
    rng = np.random.default_rng(n)
    state = {"id": np.arange(n, dtype=np.uint64)}
    for key in kpt.SYSTEM_DOUBLE_FIELDS:
        state[key] = np.zeros(n)
    for key in kpt.SYSTEM_INT_FIELDS:
        state[key] = np.zeros(n, dtype=np.int32)
    state["x"] = rng.uniform(data["x_edges"][0], data["x_edges"][-1], n)
    state["y"] = rng.uniform(data["y_edges"][0], data["y_edges"][-1], n)
    state["p"] = rng.choice(data["start_p"][data["start_p"] > 0.0], n)
    state["mu"] = rng.uniform(-0.95, 0.95, n)
    state["w"] = np.ones(n)
    return state


def _system(ctx, state, pick=slice(None)):
    part = {k: np.ascontiguousarray(v[pick]) for k, v in state.items()}
    system = ctx.system(part["id"].size, part["id"].size)
    system.upload(part)
    return system


@pytest.mark.parametrize("precision", ["f64", "mixed"])
@pytest.mark.parametrize("kind", ["parker", "focus"])
@pytest.mark.parametrize("n", SIZES)
def test_step_of_any_size(ctx, kpt, kind, precision, n):
    data = load_golden(f"lib_{kind}_readme_periodic.npz")
    grid = lib_grid(ctx, data)
    if kind == "focus":
        solver = ctx.focus_solver(grid, data["basis"], bool(data["constant_ratio"]),
                                  float(data["courant"]), float(data["spectral_index"]),
                                  float(data["h0"]), maximum_mu=float(data["max_mu"]))
    else:
        solver = ctx.parker_solver(grid, data["basis"], bool(data["constant_ratio"]),
                                   float(data["courant"]))
    solver.set_precision(kpt.PRECISION_F64 if precision == "f64" else kpt.PRECISION_MIXED)
    state = _state(kpt, data, n)

    whole = _system(ctx, state)
    dt = solver.compute_time_step(whole)
    assert dt > 0.0
    if n > 1:
        halves = [_system(ctx, state, s) for s in (slice(0, n // 2), slice(n // 2, n))]
        assert dt == min(solver.compute_time_step(h) for h in halves)
        for h in halves:
            h.close()

    none = dict(state, status=np.full(n, 2, dtype=np.int32))
    idle = _system(ctx, none)
    with pytest.raises(kpt.KptError, match="not positive and finite"):
        solver.advance_stochastic(idle, 1, 0)
    idle.close()

    again = _system(ctx, state)
    dts = [solver.advance_stochastic(again, 7, 2 + k) for k in range(3)]
    assert dts[0] == dt
    replayed = solver.advance_stochastic_steps(whole, 7, 2, 3)
    assert np.array_equal(np.asarray(replayed), np.asarray(dts))
    got, want = whole.download(), again.download()
    for key in want:
        assert np.array_equal(got[key], want[key]), key
    for h in (solver, whole, again, grid):
        h.close()
