"""Collecting a hash aggregate's groups on the device (compaction, key order,
dense columns) against numpy, at the sizes where a path or a tile ends: keys
are compared in tiles of 256 or sorted by chunks of 2048, and past 2^19 slots
sorted digit by digit, skipping digits no two keys differ in."""
import gc

import numpy as np
import pytest

from gpudbmetalcodegen_b200 import Context

pytestmark = pytest.mark.gpu

I64 = np.iinfo(np.int64)


@pytest.fixture(scope="module")
def ctx():
    with Context(0) as c:
        yield c


def make_keys(kind, n, rng):
    if kind == "dense":  # few differing digits
        return np.arange(n, dtype=np.int64) + 7
    k = rng.integers(I64.min, I64.max, size=n + 16, dtype=np.int64)  # every digit differs, both signs
    k = np.unique(np.concatenate([k[k != -1], [I64.min, I64.max]]))  # -1 is the empty-slot word
    return rng.permutation(k)[:n] if n > 2 else np.array([I64.max, I64.min])[:n]


@pytest.mark.parametrize("kind", ["dense", "mixed"])
@pytest.mark.parametrize("groups", [1, 2, 31, 255, 256, 257, 4099, 16383, 16384, 16385, 20479, 20480, 20481, 300_007])
def test_groups_come_back_in_key_order(ctx, kind, groups):
    rng = np.random.default_rng(groups)
    keys = make_keys(kind, groups, rng)
    rows = np.concatenate([keys, rng.choice(keys, size=2 * groups + 5)])
    vals = rng.integers(-10**12, 10**12, size=rows.size, dtype=np.int64)
    order = rng.permutation(rows.size)
    rows, vals = rows[order], vals[order]
    ctx.upload_table("zprobe", {"z_key": rows, "z_value": vals})
    ctx.register_symbol("zgroups", groups)
    uk, inv, cnt = np.unique(rows, return_inverse=True, return_counts=True)
    sums = np.zeros(uk.size, dtype=np.int64)
    np.add.at(sums, inv, vals)
    for tune in ("", "layout=packed"):
        got, _ = ctx.run("template=groupby", tune, arrays=True)
        assert np.array_equal(got["key"], uk) and np.array_equal(got["count"], cnt)
        assert np.array_equal(got["sum"], sums)


def test_column_arrays_outlive_the_context_and_each_other(ctx):
    """The arrays of one result share its memory: each stays valid while any
    of them lives, past later runs and past the context."""
    n = 50_000
    with Context(0) as c:
        c.upload_table("zprobe", {"z_key": np.arange(n, dtype=np.int64), "z_value": np.arange(n, dtype=np.int64) * 3})
        c.register_symbol("zgroups", n)
        key = c.run("template=groupby", arrays=True)[0]["key"]
        sums = [c.run("template=groupby", arrays=True)[0]["sum"] for _ in range(3)]
    gc.collect()
    assert np.array_equal(key, np.arange(n))
    for s in sums:
        assert np.array_equal(s, np.arange(n) * 3)
        s += 1  # an array of the caller's own
    assert np.array_equal(key, np.arange(n))


def test_unmatched_build_keys_are_no_groups(ctx):
    build = np.arange(40_000, dtype=np.int64)
    probe = np.arange(0, 40_000, 3, dtype=np.int64)
    ctx.upload_table("zbuild", {"zb_key": build, "zb_payload": (build % 1000 - 500).astype(np.int32)})
    ctx.upload_table("zprobe", {"z_key": probe, "z_value": probe})
    got, _ = ctx.run("template=hashjoin", arrays=True)
    assert np.array_equal(got["key"], probe) and (got["count"] == 1).all()
    assert np.array_equal(got["sum"], probe % 1000 - 500)
