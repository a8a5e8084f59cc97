"""The batch's choice of cell records (KPT_RECORDS_AUTO).

Populations that fill the chip on tables of more points than particles, with
fixed steps on both sides of the rule (few substeps: point tables; many:
records) and with adaptive steps: every particle ends bit for bit where the
point-table batch leaves it, over two intervals and a replayed graph.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("focused", [False, True])
@pytest.mark.parametrize("substeps", [5, 80, 0])  # 0: adaptive
def test_auto_batch_equals_point_tables(ctx, kpt, binding, fields_mod, focused, substeps):
    params = binding.default_params(kperp_over_kpara=0.05, focused=int(focused))
    settings = kpt.settings_from_dict(params)
    if substeps:
        settings.dt_min_rel = settings.dt_max_rel = (1.0 + 1e-6) / substeps
    else:
        settings.dt_min_rel = settings.dt_max_rel = 0.02
        settings.dt_min_rel = 0.01
    kind = kpt.TABLE_FOCUSED21 if focused else kpt.TABLE_PARKER16
    shapes = ((256, 512, 70001), (300, 700, 60000))
    ends = []
    try:
        for mode in (kpt.RECORDS_OFF, kpt.RECORDS_AUTO):
            ctx.set_cell_records(mode)
            batch = ctx.batch()
            handles = []
            for k, (nx, ny, n) in enumerate(shapes):
                field = fields_mod.harris_field(nx, ny, island_amplitude=0.1, noise=0.02, seed=k)
                table = ctx.field(field, kind, kpt.PRECISION_MIXED)
                parts = ctx.particles(n)
                ctx.inject(parts, table, settings, n, 4, 17 + k)
                batch.add_run(parts, table, table, settings, 17 + k, 4)
                handles.append((parts, table))
            batch.run(2)
            ends.append([h[0].download() for h in handles])
            batch.close()
            for h in handles:
                for x in h:
                    x.close()
    finally:
        ctx.set_cell_records(kpt.RECORDS_AUTO)
    for a, b in zip(*ends):
        for name in a:
            assert np.array_equal(a[name], b[name]), name
