"""Results read in one call and under the run's own wait: the same values as
the cell-by-cell entry points give, for every kind of column and for sums
beyond 64 bits; stale staged copies never reach a later answer; a context is
freed with its last reference."""
import ctypes as C
import weakref

import numpy as np
import pytest

from gpudbmetalcodegen_b200 import Context, _lib
from gpudbmetalcodegen_b200 import workloads as W
from oracle import oracle_py as O

pytestmark = pytest.mark.gpu


def cells(ctx, q):
    """The last run's result through gpudb_result_get_*."""
    lib = _lib.load()
    res = C.c_void_p()
    _lib.check(lib.gpudb_query_collect(ctx.handle, q.handle, C.byref(res)), ctx.handle)
    nc, nr = C.c_int(), C.c_longlong()
    lib.gpudb_result_shape(res, C.byref(nc), C.byref(nr))
    rows = []
    for r in range(nr.value):
        row = []
        for c in range(nc.value):
            name, t = C.create_string_buffer(64), C.c_int()
            lib.gpudb_result_column(res, c, name, 64, C.byref(t))
            if t.value == 0:
                lo, hi = C.c_int64(), C.c_int64()
                lib.gpudb_result_get_int(res, r, c, C.byref(lo), C.byref(hi))
                row.append((hi.value << 64) | (lo.value & (2**64 - 1)))
            elif t.value == 1:
                v = C.c_double()
                lib.gpudb_result_get_f64(res, r, c, C.byref(v))
                row.append(v.value)
            else:
                lib.gpudb_result_get_str(res, r, c, name, 64)
                row.append(name.value.decode())
        rows.append(tuple(row))
    text = [_lib.get_string(lib.gpudb_result_canonical, res, e) for e in (0, 1)]
    lib.gpudb_result_free(res)
    return rows, text


@pytest.mark.parametrize("scale", [1, -(3 * 10**4)])  # the second: 128-bit sums of blocks that fit 64
def test_text_and_cells_agree(scale):
    t = W.gen_fact(30_011, seed=2)
    t["f_price"] = t["f_price"] * scale
    d, p = W.gen_dim(3000, seed=2), W.gen_probe(12_000, dim_rows=3000, seed=2)
    with Context(0) as ctx:
        for name, cols in (("fact", t), ("dim", d), ("probe", p)):
            ctx.upload_table(name, cols)
        for spec in ("template=q1", "template=q1;ship_le=-1", "template=q6", "template=join_topk;k=32",
                     "template=join_topk;od_lt=0", "template=histogram", "template=anti_join", "template=join_rows"):
            q = ctx.prepare(spec)
            res, timing = ctx.run(q)
            rows, (canonical, exact) = cells(ctx, q)
            order = sorted if "rows" in spec else list  # materialised rows come in no order
            assert order(res.rows) == order(rows), spec
            assert res.canonical == canonical and res.exact == exact
            assert len(timing.phase_ms) == timing.launches and all(ms > 0 for ms in timing.phase_ms)
            assert timing.total_ms >= max(timing.phase_ms)
        if scale < 0:
            wide = ctx.run("template=q1")[0].column("sum_charge")
            assert min(wide) < -(2**63)
            assert [r[c] for r in O.q1(t) for c in ("sum_charge",)] == wide


def test_alternating_queries_keep_their_own_answers():
    t = W.gen_fact(20_000, seed=4)
    with Context(0) as ctx:
        ctx.upload_table("fact", t)
        want = {lt: O.q6(t, 0, lt, 0, 10, 51) for lt in (100, 2000, 0)}
        for graphs in (False, True):
            ctx.set_use_graphs(graphs)
            for _ in range(3):
                for lt, v in want.items():
                    spec = f"template=q6;ship_ge=0;ship_lt={lt};disc_lo=0;disc_hi=10;qty_lt=51"
                    assert ctx.run(spec, measured=2)[0].rows == [(v,)]
                    ctx.run(spec, collect=False)
                    ctx.enqueue(spec)
                    ctx.sync()
                    assert ctx.collect(ctx.prepare(spec)).rows == [(v,)]


def test_a_context_is_freed_with_its_last_reference():
    ctx = Context(0)
    ctx.upload_table("fact", W.gen_fact(100, seed=1))
    q = ctx.prepare("template=q6")
    ctx.run(q)
    gone = weakref.ref(ctx)
    assert q.ctx is ctx
    del ctx
    assert gone() is None and q.ctx is None
    assert "phase 0" in q.plan  # a query still held stays readable
