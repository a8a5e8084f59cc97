"""The page-locked pool behind downloads, on the host with a stand-in for the
library's allocator: reuse, the bound, blocks that outlive their context, and
arrays that never share memory."""
from __future__ import annotations

import ctypes
import gc
import threading

import numpy as np
import pytest


class _FakeLibrary:
    def __init__(self):
        self.live, self.allocations, self.fail = {}, 0, False

    def kpt_host_alloc(self, size, out):
        if self.fail:
            return -1
        buf = ctypes.create_string_buffer(size)
        self.live[ctypes.addressof(buf)] = buf
        self.allocations += 1
        out._obj.value = ctypes.addressof(buf)
        return 0

    def kpt_host_free(self, ptr):
        del self.live[ptr]
        return 0


@pytest.fixture()
def pool(kpt, monkeypatch):
    fake = _FakeLibrary()
    monkeypatch.setattr(kpt, "load_library", lambda: fake)
    p = kpt._PinnedPool()
    p.open()
    p.fake = fake
    return p


def test_blocks_are_reused_and_freed_with_the_last_user(pool):
    a = pool.take(3 << 20)
    a[:] = 7
    view = a[16:1024].view(np.float64)
    del a
    gc.collect()
    assert len(pool._idle) == 0  # the view still uses the block
    del view
    gc.collect()
    assert len(pool._idle) == 1
    b = pool.take(2 << 20)
    assert pool.fake.allocations == 1 and len(pool._idle) == 0
    pool.close()
    assert len(pool.fake.live) == 1  # in use
    del b
    gc.collect()
    assert len(pool.fake.live) == 0 and pool._total == 0


def test_bound_and_failures(pool):
    pool.LIMIT = 8 << 20
    held = [pool.take(3 << 20) for _ in range(3)]
    assert held[2] is None and pool._total == 6 << 20
    assert pool.take(100) is None  # small: ordinary memory
    del held
    gc.collect()
    big = pool.take(7 << 20)  # idle blocks make room
    assert big is not None and pool._total <= pool.LIMIT
    del big
    gc.collect()
    pool._trim(0)
    pool.fake.fail = True
    assert pool.take(1 << 20) is None and pool._total == 0


def test_threads_never_share_a_block(pool):
    errors = []

    def work(tag):
        for _ in range(200):
            a = pool.take(1 << 20)
            a[:4096] = tag
            if not np.all(a[:4096] == tag):
                errors.append(tag)
            del a
    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors and pool._total <= pool.LIMIT


@pytest.mark.gpu
def test_downloads_keep_their_values(ctx):
    system = ctx.system(40000, 40000)
    data = system.download()
    rng = np.random.default_rng(1)
    kept = []
    for _ in range(3):
        for key in ("x", "y", "p"):
            data[key] = rng.standard_normal(40000)
        system.upload(data)
        kept.append((data["x"].copy(), system.download()))
        data = {k: v.copy() for k, v in kept[-1][1].items()}
    for x, got in kept:
        assert np.array_equal(got["x"], x) and got["x"].flags.writeable
