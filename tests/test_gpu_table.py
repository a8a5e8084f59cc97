"""The tiled table kernel against the oracle's tables, bit for bit.

Sizes around a tile of 32 x 8 ghosted points and axes of one, two and three
cells (no derivative, only one-sided stencils, one inner point); uniform and
stretched axes; constant cells (zero slopes of either sign) and magnitudes
whose quotients leave the range of the reciprocal form.  The mixed table is
the FP64 one rounded.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = ((1, 1), (1, 9), (2, 3), (3, 2), (27, 3), (28, 4), (29, 5), (60, 12), (61, 13), (7, 70))


@pytest.mark.parametrize("scale", [1.0, 1e-150, 1e150])
@pytest.mark.parametrize("stretched", [False, True])
@pytest.mark.parametrize("nx,ny", SHAPES)
def test_table_is_the_oracles(ctx, kpt, oracle, fields_mod, nx, ny, stretched, scale):
    rng = np.random.default_rng(100 * nx + ny)
    xe, ye = np.linspace(0.0, 2.0, nx + 1), np.linspace(-1.0, 1.5, ny + 1)
    if stretched:
        xe = np.cumsum(np.concatenate([[-0.3], rng.uniform(0.5, 1.5, nx)]))
        ye = np.cumsum(np.concatenate([[0.1], rng.uniform(0.5, 1.5, ny)]))
    b, v = scale * rng.normal(size=(2, 3, ny, nx))
    b[1, : ny // 2] = 0.25 * scale
    v[0, :, : nx // 2] = -0.0
    field = fields_mod.CompactField(xe, ye, b, v)
    for focused, kind in ((False, kpt.TABLE_PARKER16), (True, kpt.TABLE_FOCUSED21)):
        want = oracle.table(field, focused=focused)
        got = ctx.field(field, kind, kpt.PRECISION_F64).table()
        assert np.array_equal(got, want)
        assert np.array_equal(np.signbit(got), np.signbit(want))
        with np.errstate(over="ignore"):
            want = want.astype(np.float32).astype(np.float64)
        assert np.array_equal(ctx.field(field, kind, kpt.PRECISION_MIXED).table(), want)
