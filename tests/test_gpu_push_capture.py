"""A push captured into a CUDA graph by the caller: capturing needs no earlier
push, and a replay is the push of the tables it was captured with, whatever
pair the context's cell records hold by then."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# thin and dense populations of a 1024 x 1024 table, both on records (AUTO)
COUNTS = (253628, 300000)


@pytest.mark.parametrize("count", COUNTS)
@pytest.mark.parametrize("warm", [False, True])  # the pair's records exist already
def test_replay_keeps_its_tables(kpt, fields_mod, count, warm):
    torch = pytest.importorskip("torch")
    settings = kpt.default_settings(kperp_over_kpara=0.05, dt_min_rel=0.005, dt_max_rel=0.005)
    rng = np.random.default_rng(count)
    names = ("x", "y", "p", "t", "step_dt", "weight", "mu")
    start = torch.zeros((7, count), dtype=torch.float64)
    start[0] = torch.from_numpy(rng.uniform(-1.0, 1.0, count))
    start[1] = torch.from_numpy(rng.uniform(-2.0, 2.0, count))
    start[2] = 0.1 * torch.from_numpy(np.exp(rng.uniform(-0.3, 0.7, count)))
    start = start.cuda()
    state = torch.zeros_like(start)
    ints = torch.zeros((2, count), dtype=torch.int32, device="cuda")
    stream = torch.cuda.Stream()
    with kpt.Context(0) as ctx, torch.cuda.stream(stream):
        ctx.set_stream(stream.cuda_stream)
        tables = [ctx.field(fields_mod.harris_field(1024, 1024, noise=0.01, seed=k),
                            kpt.TABLE_PARKER16, kpt.PRECISION_MIXED) for k in range(2)]
        ptrs = {k: state[i].data_ptr() for i, k in enumerate(names)}
        ptrs |= {"status": ints[0].data_ptr(), "split_level": ints[1].data_ptr()}
        parts = ctx.wrap_particles(count, count, ptrs)

        def push(table):
            kpt._check(ctx.lib.kpt_push_interval(ctx.handle, parts.handle, table.handle,
                                                 table.handle, ctypes.byref(settings), 0, 7, None))

        ends = []
        for table in tables:  # each table's end, on the point tables
            ctx.set_cell_records(kpt.RECORDS_OFF)
            state.copy_(start)
            push(table)
            ends.append(state.clone())
        ctx.set_cell_records(kpt.RECORDS_AUTO)
        assert not torch.equal(*ends)
        if warm:
            push(tables[0])
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        graph.capture_begin()
        push(tables[0])
        graph.capture_end()
        for other in (tables[1], tables[0], tables[1]):
            state.copy_(start)
            push(other)  # the records now hold the other table
            assert torch.equal(state, ends[tables.index(other)])
            state.copy_(start)
            graph.replay()
            assert torch.equal(state, ends[0])
        stream.synchronize()
        for h in [parts, *tables]:
            h.close()
