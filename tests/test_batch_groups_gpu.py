"""The batched group-by's tables where their forms meet: key domains at the
ends of the direct shared table (both signs, then non-negative keys only) and
of the dense global one, keys of either sign, skew, every strategy, and row
counts around a work item; each against numpy."""
import numpy as np
import pytest
import torch

from gpudbmetalcodegen_b200 import batch as B

pytestmark = pytest.mark.gpu

DIRECT = 40 * 1024 // 3  # slots of a 1,024-thread block's direct table


def run(keys, filt, vals, card, groups, mode, thr, tmpl="groupby", key_min=0, k=10, **tuning):
    cols = {n: torch.from_numpy(a).cuda() for n, a in (("k", keys), ("f", filt), ("v", vals))}
    b = B.Batch()
    if tuning:
        b.set_tuning(**tuning)
    s = B.BatchQueryStruct(tmpl=B.TPL[tmpl], thr=thr, card=card, k=k, rows=keys.size, key=cols["k"].data_ptr(),
                           filter=cols["f"].data_ptr(), value=cols["v"].data_ptr(), groups=groups, agg_mode=mode,
                           key_min=key_min, key_max=int(keys.max(initial=0)))
    b.set_queries([s])
    for _ in range(2):
        _, err = b.execute()
    rows, packed, _ = b.collect()
    n, groups_api = int(rows[0]), b.result_groups(0)
    b.close()
    return int(err[0]), packed[:n].copy(), groups_api


def expected(keys, filt, vals, card, thr):
    m = filt < thr
    r = np.fmod(keys[m].astype(np.int64), card)
    uk, inv, cnt = np.unique(r, return_inverse=True, return_counts=True)
    s = np.zeros(uk.size, np.int64)
    np.add.at(s, inv, vals[m])
    return np.stack([uk, cnt, s], axis=1)


@pytest.mark.parametrize("mode", [B.AGG_SHARED, B.AGG_GLOBAL_WARP, B.AGG_GLOBAL, B.AGG_SHARED_DIRECT])
@pytest.mark.parametrize("card", [1, 2, 7, 1024, (DIRECT + 1) // 2, (DIRECT + 1) // 2 + 1, DIRECT, DIRECT + 1, 40_003])
@pytest.mark.parametrize("sign", ["plus", "both"])
def test_domains_around_the_tables_ends(card, mode, sign):
    rng = np.random.default_rng(card)
    n = 70_001
    keys = rng.integers(-(2**31) if sign == "both" else 0, 2**31 - 1, size=n).astype(np.int32)
    keys[rng.random(n) < 0.2] = 5  # a hot key
    filt = rng.integers(0, 100, size=n).astype(np.int32)
    vals = rng.integers(-2**40, 2**40, size=n)
    want = expected(keys, filt, vals, card, 60)
    # exact groups (a hash table unless the domain fits it) and the whole domain (dense)
    for groups, tuning in ((len(want), {}), (2 * card, {}), (2 * card, dict(block=256, group_rows=4))):
        err, got, api = run(keys, filt, vals, card, groups, mode, 60, key_min=int(keys.min()), **tuning)
        assert err == 0
        assert np.array_equal(got[np.argsort(got[:, 0])], want)
        o = np.argsort(api[0])
        assert np.array_equal(np.stack([a[o] for a in api], axis=1), want)


@pytest.mark.parametrize("rows", [0, 1, 31, 33, 1023, 2049, 4096, 4097, 3_000_000])
@pytest.mark.parametrize("card", [300, 5000, 2_000_000])
def test_rows_around_work_items_and_enough_rows_for_a_direct_table(rows, card):
    rng = np.random.default_rng(rows)
    keys = (rng.zipf(1.3, size=rows) % 2**31).astype(np.int32)
    filt = rng.integers(0, 100, size=rows).astype(np.int32)
    vals = rng.integers(1, 10**6, size=rows)
    want = expected(keys, filt, vals, card, 37)
    for mode in (B.AGG_SHARED, B.AGG_SHARED_DIRECT, B.AGG_GLOBAL):
        err, got, _ = run(keys, filt, vals, card, max(1, len(want)), mode, 37)
        assert err == 0 and np.array_equal(got[np.argsort(got[:, 0])], want)


@pytest.mark.parametrize("groups", [1, 9, 16383, 16384, 16385, 70_000])
def test_top_k_over_chunks_of_the_table(groups):
    rng = np.random.default_rng(groups)
    keys = rng.permutation(np.tile(np.arange(groups, dtype=np.int32), 2))
    vals = rng.integers(-50, 50, size=keys.size)  # many ties: the key decides
    filt = np.zeros(keys.size, np.int32)
    e = expected(keys, filt, vals, 1 << 20, 1)
    e = e[np.lexsort((e[:, 0], -e[:, 2]))][:16]
    err, got, _ = run(keys, filt, vals, 1 << 20, groups, B.AGG_GLOBAL, 1, tmpl="topk", k=16)
    assert err == 0 and np.array_equal(got[:, :2], e[:, [0, 2]])
