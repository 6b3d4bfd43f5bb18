"""Sums kept as (low, high) 32-bit words in shared memory: carries, borrows
(negative values) and wrap-around must leave the exact 64-bit sum, whatever
the group count, with and without warp aggregation; and the sorted group-by
lists every created group however many a block creates."""
import numpy as np
import pytest

from gpudbmetalcodegen_b200 import Context
from oracle import oracle_py as O
from gpudbmetalcodegen_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    with Context(0) as c:
        yield c


def grouped(keys, vals):
    uk, inv, cnt = np.unique(keys, return_inverse=True, return_counts=True)
    s = np.zeros(uk.size, dtype=np.int64)
    with np.errstate(over="ignore"):
        np.add.at(s, inv, vals)
    return uk, cnt, s


@pytest.mark.parametrize("tune", ["", "warp=0", "warp=1", "warp=0;smem=11;sprobe=4;stages=2", "warp=0;layout=packed"])
@pytest.mark.parametrize("groups", [1, 3, 700, 5000])
@pytest.mark.parametrize("span", ["carry", "signed", "wrap"])
def test_groupby_sums_are_exact(ctx, tune, groups, span):
    rng = np.random.default_rng(groups)
    n = 60_001
    keys = rng.integers(0, groups, size=n, dtype=np.int64) * 1_000_003 - 5
    lo, hi = {"carry": (2**31, 2**33), "signed": (-2**40, 2**40), "wrap": (-2**62, 2**62)}[span]
    vals = rng.integers(lo, hi, size=n, dtype=np.int64)
    ctx.upload_table("zprobe", {"z_key": keys, "z_value": vals})
    ctx.register_symbol("zgroups", groups)
    got, _ = ctx.run("template=groupby", tune, arrays=True)
    uk, cnt, s = grouped(keys, vals)
    assert np.array_equal(got["key"], uk) and np.array_equal(got["count"], cnt) and np.array_equal(got["sum"], s)


@pytest.mark.parametrize("tune", ["", "keyed=2", "keyed=2;bs=256"])
def test_keyed_sums_in_shared_memory(ctx, tune):
    t = W.gen_fact(50_021, seed=6)
    t["f_price"][::7] *= -30_000  # wide sums through both words, either sign
    ctx.upload_table("fact", t)
    res, _ = ctx.run("template=q1", tune)
    for g, e in zip(res.as_dicts(), O.q1(t)):
        for k in O.Q1_AGGS:
            assert g[k] == e[k], k


@pytest.mark.parametrize("groups", [1, 5, 2047, 2048, 2049, 4096, 4097, 70_001, 700_001])
@pytest.mark.parametrize("ties", [False, True])
def test_every_group_comes_back_sorted(ctx, groups, ties):
    """Ragged group counts; with `ties` every sum is the same few values, so
    the key decides (runs of equal sums up to the whole answer)."""
    rng = np.random.default_rng(groups)
    keys = np.concatenate([np.arange(groups), rng.integers(0, groups, size=groups // 2)]).astype(np.int64)
    keys = rng.permutation(keys * 7 - 7 * (groups // 2))  # either sign, never the reserved key -1
    vals = np.ones(keys.size, np.int64) if ties else rng.integers(-10**9, 10**9, size=keys.size, dtype=np.int64)
    ctx.upload_table("zprobe", {"z_key": keys, "z_value": vals})
    ctx.register_symbol("zgroups", groups)
    uk, cnt, s = grouped(keys, vals)
    o = np.lexsort((uk, -s))
    for _ in range(2):  # twice through the same buffers
        got, t = ctx.run("template=groupby_sorted", arrays=True)
        assert t.device_error == 0
        assert np.array_equal(got["key"], uk[o]) and np.array_equal(got["count"], cnt[o])
        assert np.array_equal(got["sum"], s[o])
