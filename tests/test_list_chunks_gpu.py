"""Lists that blocks fill past their own buffers, a warp's chunk of positions
at a time: every joined row and every created group must be listed exactly
once, from no overflow through partly used chunks to blocks of many chunks."""
import numpy as np
import pytest

from gpudbmetalcodegen_b200 import Context
from oracle import oracle_py as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    with Context(0) as c:
        yield c


def tables(n_dim, n_probe, share, seed):
    """Probe rows that all pass the filter, a `share` of whose keys join."""
    rng = np.random.default_rng(seed)
    dim = {"b_key": np.arange(1, n_dim + 1, dtype=np.int32), "b_order_day": np.zeros(n_dim, np.int32),
           "b_segment": (rng.random(n_dim) < share).astype(np.uint8)}
    probe = {"p_fk": rng.integers(1, n_dim + 1, size=n_probe).astype(np.int32),
             "p_ship_day": np.full(n_probe, 2000, np.int32),
             "p_price": rng.integers(1, 10_000_000, size=n_probe), "p_discount": rng.integers(0, 11, size=n_probe)}
    return dim, probe


# one block per SM and 148 SMs: 1024 buffered entries a block (two columns),
# so ~151K rows are the last that need no chunk; 65 000 rows on 1024 threads
# give single rows per lane, the odd counts leave part chunks in every warp
@pytest.mark.parametrize("tune", ["occ=1", "occ=1;bs=1024", "occ=1;bs=64;warp=0", "occ=2;vec=4;stages=2;warp=0"])
@pytest.mark.parametrize("n_probe,share", [(65_000, 1.0), (151_553, 1.0), (160_001, 1.0), (400_003, 0.5),
                                           (3_000_017, 1.0), (3_000_017, 0.37)])
def test_every_row_and_group_is_listed_once(ctx, tune, n_probe, share):
    dim, probe = tables(1_000_003, n_probe, share, n_probe)
    ctx.upload_table("dim", dim)
    ctx.upload_table("probe", probe)
    res, t = ctx.run("template=join_topk;k=32", tune)
    assert t.device_error == 0
    top, groups, _ = O.join_topk(dim, probe, k=32)
    rows = np.flatnonzero(dim["b_segment"][probe["p_fk"] - 1] == 1)
    assert int(ctx.read_buffer("jm_n", np.uint64, 1)[0]) == rows.size
    listed = ctx.read_buffer("jm_rows", np.uint32, rows.size)
    assert np.array_equal(np.sort(listed), rows)
    assert np.array_equal(ctx.read_buffer("jm_fk", np.int32, rows.size), probe["p_fk"][listed])
    assert int(ctx.read_buffer("jg_nslots", np.uint64, 1)[0]) == groups
    assert np.unique(ctx.read_buffer("jg_slotlist", np.uint32, groups)).size == groups
    assert res.rows == top
