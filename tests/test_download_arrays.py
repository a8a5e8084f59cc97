"""What a download returns: arrays that own their memory, as arrays of numpy's own
do, and page-locked ones for callers that ask."""
from __future__ import annotations

import ctypes
import gc

import numpy as np
import pytest

SHAPES = {"id": (30001, np.uint64), "x": (30001, np.float64), "status": (30001, np.int32),
          "none": (0, np.float64)}


class _FakeContext:
    def __init__(self, calls):
        self.calls = calls

    def synchronize(self):
        self.calls.append("select")


def test_new_arrays_own_their_memory(kpt):
    out = kpt._host_arrays(SHAPES)
    for name, (n, dtype) in SHAPES.items():
        a = out[name]
        assert a.shape == (n,) and a.dtype == dtype
        assert a.flags.owndata and a.flags.writeable and a.base is None
        a[:] = 1
    column = out.pop("x")
    column.resize(40000, refcheck=False)
    assert column.size == 40000 and column[30000] == 1.0 and column[30001] == 0.0


def test_a_block_is_locked_for_its_context(kpt, monkeypatch):
    """The context's device is made current before memory is locked, and only
    then; the block is reused without."""
    calls, live = [], {}

    class Library:
        def kpt_host_alloc(self, size, out):
            calls.append("alloc")
            buf = ctypes.create_string_buffer(size)
            live[ctypes.addressof(buf)] = buf
            out._obj.value = ctypes.addressof(buf)
            return 0

        def kpt_host_free(self, ptr):
            del live[ptr]
            return 0

    library = Library()
    monkeypatch.setattr(kpt, "load_library", lambda: library)
    pool = kpt._PinnedPool()
    pool.open()
    monkeypatch.setattr(kpt, "_PINNED", pool)
    ctx = _FakeContext(calls)
    out = kpt._host_arrays(SHAPES, ctx)
    assert calls == ["select", "alloc"]
    assert not out["x"].flags.owndata and out["x"].flags.writeable
    for name, (n, dtype) in SHAPES.items():
        assert out[name].shape == (n,) and out[name].dtype == dtype
    del out
    gc.collect()
    out = kpt._host_arrays(SHAPES, ctx)
    assert calls == ["select", "alloc"]
    pool.close()
    del out
    gc.collect()
    assert not live


@pytest.mark.gpu
@pytest.mark.parametrize("count", [3, 40000])
def test_downloads(ctx, binding, count):
    rng = np.random.default_rng(count)
    system = ctx.system(count, count)
    data = system.download()
    for key in ("x", "y", "p"):
        data[key][:] = rng.standard_normal(count)
    system.upload(data)
    parts = ctx.particles(count)
    start = binding.empty_particles(count)
    for key in ("x", "y", "p"):
        start[key][:] = rng.standard_normal(count)
    parts.upload(start, count)
    for store, want in ((system, data), (parts, start)):
        own, locked = store.download(), store.download(pinned=True)
        for key in own:
            assert own[key].flags.owndata
            assert np.array_equal(own[key], want[key]) and np.array_equal(locked[key], own[key])
        own.pop("x").resize(2 * count, refcheck=False)
        store.close()
