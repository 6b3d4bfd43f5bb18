"""What a run reads back in one launch: its phases' start times, the error
word and the result's small buffers, from none to more than one launch of 32."""
import ctypes as C
from pathlib import Path

import numpy as np
import pytest

from gpudbmetalcodegen_b200 import Context
from gpudbmetalcodegen_b200 import _lib
from gpudbmetalcodegen_b200 import analyzed as A
from gpudbmetalcodegen_b200 import workloads as W

pytestmark = pytest.mark.gpu

HEADER = Path(__file__).resolve().parent.parent / "gpudbmetalcodegen_b200" / "csrc" / "kernels" / "gpudb_device.cuh"


@pytest.fixture(scope="module")
def ctx():
    with Context(0) as c:
        yield c


@pytest.mark.parametrize("spec", ["template=q1", "template=join_topk", "template=groupby_sorted"])
@pytest.mark.parametrize("warmup,measured", [(0, 1), (2, 1), (0, 4), (1, 3)])
def test_phases_fill_the_run(ctx, spec, warmup, measured):
    """The phases' times are parts of one run: none negative, together the
    total (means of the same doubles, so equal to rounding)."""
    ctx.upload_table("fact", W.gen_fact(50_000, seed=1))
    ctx.upload_table("dim", W.gen_dim(5000, seed=1))
    ctx.upload_table("probe", W.gen_probe(50_000, dim_rows=5000, seed=1))
    keys = np.arange(50_000, dtype=np.int64) % 700
    ctx.upload_table("zprobe", {"z_key": keys, "z_value": keys})
    ctx.register_symbol("zgroups", 700)
    for _ in range(3):
        res, t = ctx.run(spec, warmup=warmup, measured=measured)
        assert len(t.phase_ms) == t.launches and min(t.phase_ms) > 0
        assert sum(t.phase_ms) == pytest.approx(t.total_ms, rel=1e-9)


@pytest.mark.parametrize("naggs", [1, 31, 32, 33, 70])
def test_many_result_buffers(ctx, naggs):
    fact = W.gen_fact(20_011, seed=5)
    ctx.upload_table("fact", fact)
    aq = A.AnalyzedQuery().table("fact")
    for j in range(naggs):
        aq.agg(A.SUM, aq.binary(A.MUL, aq.col("fact", "f_quantity"), aq.lit(j + 1)), f"s{j}")
    res, t = ctx.run(aq.prepare(ctx, f"sums{naggs}"))
    q = int(fact["f_quantity"].astype(np.int64).sum())
    assert t.device_error == 0
    assert res.rows == [tuple(q * (j + 1) for j in range(naggs))]


SPIN = r"""
extern "C" __global__ void spin_100us(unsigned* gpudb_err) {
    const unsigned long long t0 = gpudb_now_ns();
    for (int i = 0; i < 1000000 && gpudb_now_ns() - t0 < 100000ull; ++i) {}
}
extern "C" __global__ void spin_300us(unsigned* gpudb_err) {
    const unsigned long long t0 = gpudb_now_ns();
    for (int i = 0; i < 1000000 && gpudb_now_ns() - t0 < 300000ull; ++i) {}
}
"""


@pytest.mark.parametrize("warmup,measured", [(0, 1), (1, 3)])
def test_hand_written_kernels_are_timed(ctx, warmup, measured):
    """Kernels that write no start time: each phase lasts at least as long as
    its loop, and not as long as both."""
    lib = _lib.load()
    src = HEADER.read_text() + SPIN
    mod = C.c_void_p()
    names = (C.c_char_p * 2)(b"spin_100us", b"spin_300us")
    _lib.check(lib.gpudb_compile(ctx.handle, src.encode(), names, 2, C.byref(mod)), ctx.handle)
    bind = (_lib.BindingDesc * 1)(_lib.BindingDesc(b"gpudb_err", _lib.PARAM_ERROR_WORD, b"unsigned", None, None, 1, 0, 0))
    ph = (_lib.PhaseDesc * 2)(*(_lib.PhaseDesc(n, None, 32, 1, 0, 0, 0, 1, bind, 1) for n in names))
    t = _lib.Timing()
    _lib.check(lib.gpudb_execute(ctx.handle, mod, ph, 2, 0, 2, warmup, measured, C.byref(t)), ctx.handle)
    lib.gpudb_module_free(mod)
    assert 0.1 <= t.phase_ms[0] < 0.3 <= t.phase_ms[1] < 0.4
    assert t.phase_ms[0] + t.phase_ms[1] == pytest.approx(t.total_ms, rel=1e-9)
