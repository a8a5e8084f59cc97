"""A batch whose stores grow, shrink or are sorted on their own between two
runs of the same loop: the replayed graph must follow (bit for bit the runs
pushed without a graph)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = ((24, 40, 700), (32, 64, 1500))  # nx, ny, capacity


def _start(binding, capacity, seed):
    rng = np.random.default_rng(seed)
    start = binding.empty_particles(capacity)
    start["x"][:] = rng.uniform(-1.0, 1.0, capacity)
    start["y"][:] = rng.uniform(-2.0, 2.0, capacity)
    start["p"][:] = 0.1 * np.exp(rng.uniform(-0.3, 0.7, capacity))
    start["w"][:] = 1.0
    start["mu"][:] = rng.uniform(-0.9, 0.9, capacity)
    start["status"][:] = 0
    return start


@pytest.mark.parametrize("focused", [False, True])
@pytest.mark.parametrize("second", [0.3, 2.0])  # the later counts, of the first
def test_replay_follows_the_counts(ctx, kpt, fields_mod, binding, focused, second):
    kind = kpt.TABLE_FOCUSED21 if focused else kpt.TABLE_PARKER16
    settings = kpt.default_settings(kperp_over_kpara=0.05, focused=int(focused),
                                    dt_min_rel=0.05, dt_max_rel=0.05)
    ends = []
    for use_graph in (False, True):
        batch, handles = ctx.batch(), []
        for seed, (nx, ny, capacity) in enumerate(SIZES):
            table = ctx.field(fields_mod.harris_field(nx, ny, noise=0.01, seed=seed), kind,
                              kpt.PRECISION_MIXED)
            parts = ctx.particles(capacity)
            parts.upload(_start(binding, capacity, seed), capacity // 2)
            batch.add_run(parts, table, table, settings, seed, 0)
            handles.append((parts, table))
        batch.set_schedule(sort_tile=8, blocks_per_sm=0, sort_every=1)
        batch.run(2, use_graph=use_graph)
        for seed, (parts, table) in enumerate(handles):
            count = min(int(second * (parts.count)), SIZES[seed][2])
            full = _start(binding, SIZES[seed][2], seed + 10)
            full["t"][:] = 2 * settings.mhd_dt
            parts.upload(full, count)
            if seed == 1:
                ctx.sort(parts, table, 8, 8)  # takes the store's sort buffers anew
        batch.run(2, use_graph=use_graph)
        ends.append([(h[0].count, h[0].download()) for h in handles])
        batch.close()
        for hs in handles:
            for h in hs:
                h.close()
    for (n, want), (m, got) in zip(*ends):
        assert n == m
        for name in want:
            assert np.array_equal(want[name], got[name]), name
        assert np.all(got["t"] > 2.5 * settings.mhd_dt)  # every particle was pushed
