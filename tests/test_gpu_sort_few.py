"""The tile sort on both sides of the population from which ranks are taken in
shared memory (8192 particles and 32 a word): every particle is pushed, to the same
end as unsorted."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8191, 8192, 8193, 16415, 16416, 16417])
@pytest.mark.parametrize("tile", [2, 8, 64])  # 513, 33 and 2 words
def test_both_rankings_reach_every_particle(ctx, kpt, binding, fields_mod, n, tile):
    tables = [ctx.field(fields_mod.harris_field(32, 64, noise=0.02, seed=s), kpt.TABLE_PARKER16,
                        kpt.PRECISION_MIXED) for s in (5, 6)]
    settings = kpt.settings_from_dict(binding.default_params(kperp_over_kpara=0.05))
    parts = ctx.particles(n)
    ctx.inject(parts, tables[0], settings, n, 4, 17)
    start = parts.download(n)
    start["status"][::11] = 1
    ends = []
    for ordered in (False, True):
        parts.upload(start, n)
        if ordered:
            ctx.sort(parts, tables[0], tile, tile)
        stats = ctx.push_interval(parts, *tables, settings, 4, 17)
        ends.append((stats.particle_steps, parts.download(n)))
    for h in (parts, *tables):
        h.close()
    assert ends[0][0] == ends[1][0] > 0
    for name in ends[0][1]:
        assert np.array_equal(ends[0][1][name], ends[1][1][name]), name
