"""A small table's groups are collected right behind its kernels: repeated,
warmed-up, uncollected, failing and growing runs must each return their own
groups. Up to 2^14 slots (8192 groups at load 1/2) keys are compared in tiles
of 256, up to 2^19 they are sorted by chunks of 2048; larger tables are
collected after the run, by radix passes over tiles of 1024."""
import numpy as np
import pytest

from gpudbmetalcodegen_b200 import Context
from gpudbmetalcodegen_b200._lib import GpudbError

pytestmark = pytest.mark.gpu


def load(ctx, keys, scale):
    ctx.upload_table("zprobe", {"z_key": keys, "z_value": keys * scale})


def check(got, keys, scale):
    uk, cnt = np.unique(keys, return_counts=True)
    assert np.array_equal(got["key"], uk) and np.array_equal(got["count"], cnt)
    assert np.array_equal(got["sum"], uk * cnt * scale)


@pytest.mark.parametrize("tune", ["", "layout=packed"])
@pytest.mark.parametrize("groups", [1, 255, 256, 257, 4097, 8192, 8193, 10_240, 131_073, 262_144, 262_145, 263_168, 300_007])
def test_each_run_returns_its_own_groups(groups, tune):
    rng = np.random.default_rng(groups)
    with Context(0) as ctx:
        ctx.register_symbol("zgroups", groups)
        kept = []
        for i in range(4):
            keys = rng.permutation(np.arange(3 * groups, dtype=np.int64) % groups) * (-0x2545F4914F6CDD1) + i
            load(ctx, keys, i + 1)
            if i == 2:
                ctx.run("template=groupby", tune, collect=False)
            got, t = ctx.run("template=groupby", tune, arrays=True, warmup=i % 2, measured=1 + i % 3)
            assert t.device_error == 0
            kept.append((got, keys, i + 1))
        for k in kept:  # the earlier answers are still their own
            check(*k)


def test_a_failed_run_returns_nothing_and_the_next_one_its_own():
    with Context(0) as ctx:
        ctx.register_symbol("zgroups", 10)
        keys = np.arange(40_000, dtype=np.int64)  # more groups than the table has slots
        load(ctx, keys, 1)
        with pytest.raises(GpudbError):
            ctx.run("template=groupby", arrays=True)
        keys = keys % 9
        load(ctx, keys, 3)
        check(ctx.run("template=groupby", arrays=True)[0], keys, 3)


@pytest.mark.parametrize("groups", [700, 70_001])
def test_replayed_graphs_return_the_same_groups(groups):
    """Captured fills, kernels and, for the sorted form, a cooperative sort."""
    keys = np.random.default_rng(5).permutation(np.arange(5 * groups, dtype=np.int64) % groups) * 31
    with Context(0) as ctx:
        ctx.register_symbol("zgroups", groups)
        load(ctx, keys, 2)
        ctx.set_use_graphs(True)
        q, s = ctx.prepare("template=groupby"), ctx.prepare("template=groupby_sorted")
        for _ in range(4):
            check(ctx.run(q, arrays=True)[0], keys, 2)
            got, t = ctx.run(s, collect=False)
            n = int(ctx.read_buffer("gss_n", np.uint64, 1)[0])
            assert t.device_error == 0 and n == groups
            k, v = ctx.read_buffer("gss_out_k", np.int64, n), ctx.read_buffer("gss_out_v", np.int64, n)
            uk, cnt = np.unique(keys, return_counts=True)
            o = np.lexsort((uk, -(uk * cnt * 2)))
            assert np.array_equal(k, uk[o]) and np.array_equal(v, (uk * cnt * 2)[o])
