"""The check of a host field's cells, made by the table kernel.

A cell with an infinity or NaN in any component of B or V is refused with the
reader's message, wherever it lies (corners, rows and columns that only their
own thread reads, a field of one cell) and in every kind of table; the largest
finite values are accepted.  A bad cell is reported ahead of a bad axis, as
the cells are read first.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NX, NY = 37, 5


def _field(fields_mod, nx, ny):
    rng = np.random.default_rng(3)
    return fields_mod.CompactField(np.linspace(0.0, 2.0, nx + 1), np.linspace(-1.0, 1.0, ny + 1),
                                   rng.normal(size=(3, ny, nx)), rng.normal(size=(3, ny, nx)))


@pytest.mark.parametrize("precision", ["f64", "mixed"])
@pytest.mark.parametrize("kind", ["TABLE_PARKER16", "TABLE_FOCUSED21"])
def test_bad_cells_are_refused(ctx, kpt, fields_mod, kind, precision):
    prec = kpt.PRECISION_F64 if precision == "f64" else kpt.PRECISION_MIXED
    for nx, ny in ((NX, NY), (1, 1)):
        field = _field(fields_mod, nx, ny)
        ctx.field(field, getattr(kpt, kind), prec).close()
        cells = {(0, 0), (ny - 1, nx - 1), (ny // 2, nx // 3), (0, nx - 1)}
        for k, (j, i) in enumerate(sorted(cells)):
            for values in (field.b, field.v):
                for comp in range(3):
                    kept = values[comp, j, i]
                    values[comp, j, i] = (np.nan, np.inf, -np.inf)[(k + comp) % 3]
                    with pytest.raises(kpt.KptError, match="non-finite field value"):
                        ctx.field(field, getattr(kpt, kind), prec)
                    values[comp, j, i] = np.finfo(np.float64).max
                    ctx.field(field, getattr(kpt, kind), prec).close()
                    values[comp, j, i] = kept


def test_bad_cell_comes_before_bad_axis(ctx, kpt, fields_mod):
    field = _field(fields_mod, NX, NY)
    field.x_edges[3] = field.x_edges[2]
    with pytest.raises(kpt.KptError, match="strictly ascending"):
        ctx.field(field)
    field.v[2, NY - 1, NX - 1] = np.nan
    with pytest.raises(kpt.KptError, match="non-finite field value"):
        ctx.field(field)
