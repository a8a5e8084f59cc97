"""The tile sort of the push order.

The order is a permutation: a push in sorted order ends every particle bit
for bit where the unsorted push leaves it, and a particle left out would stay
behind.  Populations around a chunk of 512 and beyond one pass of the largest
grid, tile counts on both sides of the shared-memory ranking (2048 words), all
particles in one tile, and populations with escaped particles.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[(23, 89), (32, 64)])  # 2048 and 2049 words at tile 1
def tables(request, ctx, kpt, fields_mod):
    nx, ny = request.param
    out = [ctx.field(fields_mod.harris_field(nx, ny, island_amplitude=0.1, noise=0.02, seed=s),
                     kpt.TABLE_PARKER16, kpt.PRECISION_MIXED) for s in (5, 6)]
    yield out
    for t in out:
        t.close()


@pytest.mark.parametrize("where", ["spread", "one tile"])
@pytest.mark.parametrize("tile", [1, 8])
@pytest.mark.parametrize("n", [1, 31, 511, 512, 513, 7001, 152 * 16 * 512 + 17])
def test_sorted_push_reaches_every_particle(ctx, kpt, binding, tables, n, tile, where):
    params = binding.default_params(kperp_over_kpara=0.05)
    settings = kpt.settings_from_dict(params)
    parts = ctx.particles(n)
    ctx.inject(parts, tables[0], settings, n, 4, 17)
    start = parts.download(n)
    if where == "one tile":
        start["x"][:] = start["x"][0]
        start["y"][:] = start["y"][0]
    start["status"][::7] = 1
    ends = []
    for ordered in (False, True):
        parts.upload(start, n)
        if ordered:
            ctx.sort(parts, tables[0], tile, tile)
        stats = ctx.push_interval(parts, tables[0], tables[1], settings, 4, 17)
        ends.append((stats.particle_steps, parts.download(n)))
    parts.close()
    assert ends[0][0] == ends[1][0] and (n < 2 or ends[0][0] > 0)
    for name in ends[0][1]:
        assert np.array_equal(ends[0][1][name], ends[1][1][name]), name
