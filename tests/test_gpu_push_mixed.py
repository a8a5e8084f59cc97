"""The mixed push's builds (few particles, point tables, dense on records or
points) at the populations where the choice changes: every build leaves every
particle at the same bits, and counts the same steps."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FRAME, SEED = 5, 91


@pytest.fixture(scope="module")
def network(ctx, kpt):
    settings = kpt.default_settings(focused=1, closure=kpt.CLOSURE_SURROGATE)
    net = ctx.train_surrogate(settings, samples=20000, steps=100, batch=2048, hidden_width=32)
    yield net
    net.close()


def _push(ctx, parts, tables, settings, start, n, blocks, records, kpt):
    parts.upload(start, n)
    ctx.set_push_schedule(kpt.SCHEDULE_REFILL, blocks)
    ctx.set_cell_records(records)
    try:
        stats = ctx.push_interval(parts, tables[0], tables[1], settings, FRAME, SEED)
    finally:
        ctx.set_push_schedule(kpt.SCHEDULE_REFILL, 0)
        ctx.set_cell_records(kpt.RECORDS_AUTO)
    return parts.download(), \
        (stats.particle_steps, stats.pushed, stats.failed, stats.max_steps)


# one particle, the lane cap's steps (1216 warps of eight per SM), the last
# population of the few-particle build and the first beyond it, one that fills
# the chip
@pytest.mark.parametrize("n", [1, 1216, 1217, 38912, 38913, 125000])
@pytest.mark.parametrize("focused,learned", [(0, False), (1, False), (1, True)])
def test_builds_agree(ctx, kpt, network, n, focused, learned):
    rng = np.random.default_rng(n)
    closure = kpt.CLOSURE_SURROGATE if learned else kpt.CLOSURE_QLT
    settings = kpt.default_settings(focused=focused, closure=closure if focused else 0,
                                    max_steps=12)
    if n % 2:
        settings.dt_min_rel = settings.dt_max_rel = 1.0 / 8.0
    ye = kpt.fields.stretched_edges(90, -2.0, 2.0)
    frames = [kpt.fields.harris_field(70, 90, y_edges=ye, noise=0.02, seed=s) for s in (1, 2)]
    kind = kpt.TABLE_FOCUSED21 if focused else kpt.TABLE_PARKER16
    tables = [ctx.field(f, kind, kpt.PRECISION_MIXED) for f in frames]
    start = {"x": rng.uniform(-1.0, 1.0, n), "y": rng.uniform(-2.0, 2.0, n),
             "p": np.full(n, settings.p0), "t": np.full(n, FRAME * settings.mhd_dt),
             "dt": np.zeros(n), "w": np.ones(n), "mu": rng.uniform(-0.99, 0.99, n),
             "status": (rng.random(n) < 0.05).astype(np.int32) * (n > 1),
             "level": np.zeros(n, dtype=np.int32)}
    if learned:
        ctx.set_surrogate(network)
    parts = ctx.particles(n)
    try:
        want, counts = _push(ctx, parts, tables, settings, start, n, 0, kpt.RECORDS_OFF, kpt)
        assert counts[1] == int(np.sum(start["status"] == 0))
        for blocks, records in ((0, kpt.RECORDS_AUTO), (0, kpt.RECORDS_ON), (1, kpt.RECORDS_OFF),
                                (3, kpt.RECORDS_OFF), (4, kpt.RECORDS_OFF), (5, kpt.RECORDS_ON)):
            got, again = _push(ctx, parts, tables, settings, start, n, blocks, records, kpt)
            assert again == counts, (blocks, records)
            for key in ("x", "y", "p", "t", "dt", "mu", "status"):
                assert np.array_equal(got[key], want[key]), (key, blocks, records)
    finally:
        ctx.set_surrogate(None)
