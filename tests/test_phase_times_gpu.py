"""What a run reads back in one launch: its phases' start times, the error
word and the result's small buffers, from none to more than one launch of 32."""
import numpy as np
import pytest

from gpudbmetalcodegen_b200 import Context
from gpudbmetalcodegen_b200 import analyzed as A
from gpudbmetalcodegen_b200 import workloads as W

pytestmark = pytest.mark.gpu


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
