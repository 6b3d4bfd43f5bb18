"""What a batch and the sizer leave in pinned memory: result rows collected
twice and after other calls, refused before an execution, and predictions on
both sides of the size that crosses the link in place."""
import numpy as np
import pytest
import torch

from gpudbmetalcodegen_b200 import batch as B
from gpudbmetalcodegen_b200._lib import GpudbError

pytestmark = pytest.mark.gpu


def queries(n, rows):
    g = torch.Generator(device="cuda").manual_seed(n)
    cols = {"keys": torch.randint(0, 500, (rows,), generator=g, device="cuda", dtype=torch.int32),
            "filter": torch.randint(0, 10_000, (rows,), generator=g, device="cuda", dtype=torch.int32),
            "vals": torch.randint(-10**9, 10**9, (rows,), generator=g, device="cuda", dtype=torch.int64)}
    torch.cuda.synchronize()
    a = np.zeros(n, dtype=B.QUERY_DTYPE)
    for i in range(n):
        a[i]["tmpl"] = B.TPL[("groupby", "topk", "agg")[i % 3]]
        a[i]["rows"] = rows - i % 7
        a[i]["thr"] = 37 * i % 10_001
        a[i]["key"], a[i]["filter"], a[i]["value"] = (cols[c].data_ptr() for c in ("keys", "filter", "vals"))
        a[i]["card"], a[i]["k"], a[i]["groups"], a[i]["key_max"], a[i]["filter_max"] = 500, 5, 500, 499, 9999
    return a, {c: v.cpu().numpy() for c, v in cols.items()}, cols


def check(a, rows, packed, t):
    off = 0
    for q, r in zip(a, rows):
        blk = packed[off:off + int(r)]
        off += int(r)
        n = int(q["rows"])
        m = t["filter"][:n] < q["thr"]
        k, v = t["keys"][:n][m], t["vals"][:n][m]
        cnt, s = np.bincount(k, minlength=500), np.zeros(500, np.int64)
        np.add.at(s, k, v)
        at = np.flatnonzero(cnt)
        if q["tmpl"] == B.TPL["groupby"]:
            assert np.array_equal(blk[np.argsort(blk[:, 0])], np.stack([at, cnt[at], s[at]], 1))
        elif q["tmpl"] == B.TPL["topk"]:
            best = at[np.lexsort((at, -s[at]))][:5]
            assert np.array_equal(blk[:, :2], np.stack([best, s[best]], 1))
        else:
            assert blk[0, 0] == cnt.sum() and blk[0, 1] == s.sum()
    assert off == packed.shape[0]


@pytest.mark.parametrize("use_graph", [False, True])
@pytest.mark.parametrize("n", [1, 2, 33, 1024, 1025, 5000])
def test_collected_again_and_again(n, use_graph):
    a, t, keep = queries(n, 3001 if n > 100 else 70_001)
    b = B.Batch()
    b.set_queries(a)
    with pytest.raises(GpudbError):
        b.collect()
    for _ in range(3):
        b.execute(use_graph)
        first = b.collect()
        check(a, first[0], first[1], t)
        b.features()
        again = b.collect()
        check(a, again[0], again[1], t)
    b.close()


@pytest.mark.parametrize("n", [1, 15, 16, 17, 8191, 8192, 8193])
def test_predictions_on_both_sides_of_the_pinned_size(n):
    """A sample's outputs take the same operations in the same order on every
    path, so they are equal bit for bit."""
    X = np.random.default_rng(n).random((9000, 16), dtype=np.float32)
    s = B.Sizer(seed=3)
    assert np.array_equal(s.predict(X[:n]), s.predict(X)[:n])
    s.close()
