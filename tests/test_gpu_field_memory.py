"""Fields that do not fit in device memory: the failure leaves nothing behind for
the next call, and a non-finite cell is reported ahead of it, as the cells are
read first."""
from __future__ import annotations

import contextlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def _full_device(torch, left):
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    held = torch.empty(free - left, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del held
        torch.cuda.empty_cache()


@pytest.fixture()
def field(fields_mod):
    return fields_mod.harris_field(512, 1024, noise=0.01, seed=1)  # an FP64 table of 93 MB


def test_out_of_memory_leaves_no_error_behind(ctx, kpt, field):
    torch = pytest.importorskip("torch")
    ctx.synchronize()
    with _full_device(torch, 48 << 20):
        with pytest.raises(kpt.KptError, match="memory"):
            ctx.field(field, kpt.TABLE_FOCUSED21, kpt.PRECISION_F64)
    ctx.field(field, kpt.TABLE_FOCUSED21, kpt.PRECISION_F64).close()


def test_bad_cell_comes_before_out_of_memory(ctx, kpt, field):
    torch = pytest.importorskip("torch")
    ctx.synchronize()
    field.v[2, -1, -1] = float("inf")
    with _full_device(torch, 48 << 20):
        with pytest.raises(kpt.KptError, match="non-finite field value"):
            ctx.field(field, kpt.TABLE_FOCUSED21, kpt.PRECISION_F64)
