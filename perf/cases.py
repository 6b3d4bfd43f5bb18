"""The measured cases: queries as a program sends them to this engine.

Every case goes through the public entry points (`Context.run`,
`Context.read_buffer`, `BatchRunner.run`, `Sizer.grads`) with the default
tuning, over seeded tables that are resident in HBM, and returns the whole
answer on the host. The kinds:

  q1            scan -> filter -> six-bucket aggregate over the fact table
  q6            scan -> filter -> one exact sum over the fact table
  join          bitmap semi-join -> group-by -> top-k over dim / probe
  groupby       hash group-by, every group returned in key order
  groups_sorted hash group-by, every group returned by ORDER BY sum DESC, key;
                the columns are read into the program's own pinned arrays
  hashjoin      hash build + probe, per-key count and sum in key order
  multi_join    the five-phase snowflake join
  batch         mixed queries (agg, join, groupby, topk) as one batch, hash
                tables sized by the trained network
  sizer         forward and backward pass of that network

Table sizes and distributions are those of the engine's workloads
(gpudbmetalcodegen_b200/workloads.py, bench.py).
"""
import math

import numpy as np
import torch

from gpudbmetalcodegen_b200 import batch as B
from gpudbmetalcodegen_b200.engine import Context

FACT_CUTOFF = 1263
MIX_ZIPF = (0.8, 0.95, 1.1, 1.3)
MIX_RANKS = 1 << 22
MIX_DIM_ROWS = 1_000_000
GROUPS_READ = 1 << 16  # largest key domain whose every group a batch's client reads


def listed():
    return [
        # one interactive query on a small table: latency and launches
        {"name": "q1_small", "kind": "q1", "rows": 60_175, "ship_le": 2436},
        # the benchmark's fact table (scale factor 1), aggregate and grouping
        {"name": "q1_sf1", "kind": "q1", "rows": 6_001_215, "ship_le": 2436},
        # the selective sum at scale factor 10
        {"name": "q6_sf10", "kind": "q6", "rows": 59_986_052},
        # an ordinary small join with ragged sizes
        {"name": "join_small", "kind": "join", "dim": 150_000, "probe": 600_037, "od_lt": 1170, "ship_gt": 1170, "k": 10},
        # the benchmark's join: 15M build rows, 60M probe rows
        {"name": "join_sf10", "kind": "join", "dim": 15_000_000, "probe": 60_000_000, "od_lt": 1170, "ship_gt": 1170,
         "k": 10},
        # a report over a few thousand skewed keys, all groups collected
        {"name": "groupby_4k", "kind": "groupby", "rows": 1_000_003, "keys": 4_099, "s": 1.1},
        # the skewed-key stress at full size, every group in sum order
        {"name": "groups_sorted_120m", "kind": "groups_sorted", "rows": 120_000_000, "keys": 1 << 22, "s": 1.1},
        # a skewed-key join whose million-key answer is collected
        {"name": "hashjoin_30m", "kind": "hashjoin", "rows": 30_000_001, "keys": 1 << 20, "s": 1.1},
        # the snowflake join at its benchmark size
        {"name": "multi_join_60m", "kind": "multi_join", "cust": 1_500_000, "supp": 100_000, "orders": 15_000_000,
         "lines": 60_000_000},
        # what one serving tick admits: a few queries over slices
        {"name": "batch_tick", "kind": "batch", "queries": 4, "mix": 5, "table": 8_000_000, "min_rows": 1_000_000,
         "max_rows": 8_000_000, "max_card": 1 << 22},
        # the mixed workload: uneven slices, cardinalities up to 2^22
        {"name": "batch_mixed", "kind": "batch", "queries": 64, "mix": 7, "table": 60_000_000, "min_rows": 1_000_000,
         "max_rows": 60_000_000, "max_card": 1 << 22},
        # one full-batch pass over the network's training log
        {"name": "sizer_grads", "kind": "sizer", "rows": 100_003},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["q1", "q6", "join", "groupby", "groups_sorted", "hashjoin", "multi_join", "batch", "sizer"])
    s = rng.choice([0.0, 0.8, 0.95, 1.1, 1.3])  # 0: uniform keys
    if kind == "q1":
        return {"kind": kind, "rows": _log_int(rng, 20_000, 60_000_000), "ship_le": rng.choice([2436, 2436, 1200, 400])}
    if kind == "q6":
        return {"kind": kind, "rows": _log_int(rng, 20_000, 60_000_000)}
    if kind == "join":
        probe = _log_int(rng, 200_000, 60_000_000)
        return {"kind": kind, "dim": max(1000, int(probe * rng.uniform(0.05, 0.25))), "probe": probe,
                "od_lt": rng.choice([1170, 1170, 300, 2000]), "ship_gt": rng.choice([1170, 1170, 400, 2000]),
                "k": rng.choice([1, 10, 10, 32])}
    if kind == "groupby":
        return {"kind": kind, "rows": _log_int(rng, 100_000, 10_000_000), "keys": _log_int(rng, 16, 1 << 16), "s": s}
    if kind == "groups_sorted":
        rows = _log_int(rng, 1_000_000, 120_000_000)
        return {"kind": kind, "rows": rows, "keys": min(rows, _log_int(rng, 1 << 10, 1 << 22)), "s": s}
    if kind == "hashjoin":
        rows = _log_int(rng, 500_000, 30_000_000)
        return {"kind": kind, "rows": rows, "keys": min(rows, _log_int(rng, 1 << 8, 1 << 20)), "s": s}
    if kind == "multi_join":
        lines = _log_int(rng, 400_000, 60_000_000)
        return {"kind": kind, "cust": max(100, lines // 40), "supp": max(50, lines // 600),
                "orders": max(400, int(lines * rng.uniform(0.2, 0.25))), "lines": lines}
    if kind == "batch":
        hi = _log_int(rng, 2_000_000, 60_000_000)
        return {"kind": kind, "queries": _log_int(rng, 1, 64), "mix": rng.randrange(1, 1 << 20), "table": hi,
                "min_rows": 1_000_000, "max_rows": hi, "max_card": _log_int(rng, 1 << 10, 1 << 22)}
    return {"kind": "sizer", "rows": _log_int(rng, 300, 100_000)}


# ---------------------------------------------------------------------------
# tables, made on the GPU from the seed
# ---------------------------------------------------------------------------
class _Rng:
    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(int(seed) * 1_000_003 + 17)

    def ints(self, lo, hi, n, dtype):
        """Uniform on lo..hi, both ends included."""
        return torch.randint(lo, hi + 1, (n,), generator=self.g, device="cuda", dtype=dtype)

    def perm(self, n):
        return torch.randperm(n, generator=self.g, device="cuda")

    def ranks(self, n, keys, s):
        """Zipf(s) ranks below `keys`; s = 0 is uniform."""
        if s == 0:
            return self.ints(0, keys - 1, n, torch.int64)
        cdf = torch.arange(1, keys + 1, device="cuda", dtype=torch.float64).pow_(-s).cumsum(0)
        out = torch.empty(n, device="cuda", dtype=torch.int64)
        for a in range(0, n, 30_000_000):
            b = min(n, a + 30_000_000)
            u = torch.rand(b - a, generator=self.g, device="cuda", dtype=torch.float64) * cdf[-1]
            out[a:b] = torch.searchsorted(cdf, u, right=True).clamp_(max=keys - 1)
        return out


def _fact(case, seed):
    r, n = _Rng(seed), case["rows"]
    ship = r.ints(0, 2526, n, torch.int32)
    t = {"f_ship_day": ship, "f_quantity": r.ints(1, 50, n, torch.int64), "f_price": r.ints(90_000, 10_500_000, n, torch.int64),
         "f_discount": r.ints(0, 10, n, torch.int64), "f_tax": r.ints(0, 8, n, torch.int64)}
    returned = ship + r.ints(1, 30, n, torch.int32) <= FACT_CUTOFF
    a_or_r = torch.where(r.ints(0, 1, n, torch.int32) == 0, ord("A"), ord("R"))
    t["f_flag_a"] = torch.where(returned, a_or_r, ord("N")).to(torch.uint8)
    t["f_flag_b"] = torch.where(ship <= FACT_CUTOFF, ord("F"), ord("O")).to(torch.uint8)
    return t


def _dim_probe(case, seed):
    r, nd, n = _Rng(seed), case["dim"], case["probe"]
    key = (r.perm(nd) + 1).to(torch.int32)
    oday = r.ints(0, 2405, nd, torch.int32)
    dim = {"b_key": key, "b_order_day": oday, "b_segment": r.ints(0, 4, nd, torch.uint8)}
    by_key = torch.zeros(nd + 1, device="cuda", dtype=torch.int32)
    by_key[key.long()] = oday
    fk = r.ints(1, nd, n, torch.int32)
    probe = {"p_fk": fk, "p_ship_day": by_key[fk.long()] + r.ints(1, 121, n, torch.int32),
             "p_price": r.ints(90_000, 10_500_000, n, torch.int64), "p_discount": r.ints(0, 10, n, torch.int64)}
    return dim, probe


def _key_of_rank(keys, seed):
    """Distinct, well mixed non-negative 63-bit keys, one per rank."""
    m62 = (1 << 62) - 1
    x = torch.arange(keys, device="cuda", dtype=torch.int64) ^ (int(seed) * 0x9E3779B9 & m62)
    for c in (0x2545F4914F6CDD1D, 0x369DEA0F31A53F85):  # odd: a bijection modulo 2^62
        x = (x * c) & m62
        x = x ^ (x >> 31)
    return x


def _skewed(case, seed):
    """Skewed keys of which every one occurs (a fact row per key of the
    dimension at least), so an answer has as many groups as there are keys."""
    r = _Rng(seed)
    n, keys = case["rows"], case["keys"]
    ranks = r.ranks(n, keys, case["s"])
    ranks[torch.arange(keys, device="cuda") * n // keys] = r.perm(keys)
    return ranks, _key_of_rank(keys, seed), r


def _snowflake(case, seed):
    r = _Rng(seed)
    nc, ns, no, nl = case["cust"], case["supp"], case["orders"], case["lines"]
    i32 = torch.int32

    def seq(n):
        return torch.arange(1, n + 1, device="cuda", dtype=i32)

    nation = torch.arange(25, device="cuda", dtype=i32)
    return {"nation": {"n_key": nation, "n_region": nation % 5},
            "cust": {"c_key": seq(nc), "c_nation": r.ints(0, 24, nc, i32)},
            "supp": {"s_key": seq(ns), "s_nation": r.ints(0, 24, ns, i32)},
            "ord": {"o_key": seq(no), "o_cust": r.ints(1, nc, no, i32), "o_day": r.ints(0, 2405, no, i32)},
            "line": {"l_okey": r.ints(1, no, nl, i32), "l_supp": r.ints(1, ns, nl, i32),
                     "l_price": r.ints(90_000, 10_500_000, nl, torch.int64), "l_discount": r.ints(0, 10, nl, torch.int64)}}


def _mix_queries(case, seed):
    """The batch's shapes come from the case (so its work is known), the
    slices' tables and offsets from the seed."""
    shape, place = np.random.default_rng(case["mix"]), np.random.default_rng(int(seed))
    out = []
    for _ in range(case["queries"]):
        tmpl = B.TEMPLATES[int(shape.integers(len(B.TEMPLATES)))]
        rows = int(round(math.exp(shape.uniform(math.log(case["min_rows"]), math.log(case["max_rows"])))))
        rows = max(1, min(rows, case["table"]))
        top = min(case["max_card"], GROUPS_READ) if tmpl == "groupby" else case["max_card"]
        card = int(round(math.exp(shape.uniform(math.log(4), math.log(top)))))
        out.append(B.MixQuery(tmpl=tmpl, table=int(place.integers(len(MIX_ZIPF))),
                              row0=int(place.integers(0, case["table"] - rows + 1)), rows=rows,
                              thr=int(round(shape.uniform(0.01, 0.99) * 10_000)),
                              key="m_rank_z" if shape.random() < 0.5 else "m_rank_u", card=card, k=10,
                              attr_lt=int(shape.integers(1, 1000))))
    return out


def _mix_tables(case, seed):
    return B.MixTables(case["table"], MIX_ZIPF, MIX_RANKS, MIX_DIM_ROWS, seed=1 + int(seed))


_SIZER = []


def _trained_sizer():
    """The network a program trains once, on its own log, and keeps."""
    if not _SIZER:
        case = {"queries": 3000, "mix": 1, "table": 60_000_000, "min_rows": 500_000, "max_rows": 60_000_000,
                "max_card": MIX_RANKS}
        tables, log = _mix_tables(case, 0), B.ExecutionLog()
        B.log_executions(tables, _mix_queries(case, 0), log)
        _SIZER.append(B.train_sizer(log, epochs=150, batch=256)[0])
    return _SIZER[0]


def _sizer_data(case, seed):
    r = np.random.default_rng(int(seed))
    params = []
    for out, inp in ((64, 16), (64, 64), (64, 64), (2, 64)):
        lim = math.sqrt(6.0 / inp)
        params += [r.uniform(-lim, lim, out * inp), r.uniform(-0.05, 0.05, out)]
    return (np.concatenate(params).astype(np.float32), r.random((case["rows"], 16), dtype=np.float32),
            r.random((case["rows"], 2), dtype=np.float32))


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def _register(ctx, tables):
    for table, cols in tables.items():
        for name, t in cols.items():
            ctx.register_tensor(table, name, t)


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind, "case": case}
    if kind == "sizer":
        params, st["X"], st["Y"] = _sizer_data(case, seed)
        st["sizer"] = B.Sizer(seed=1)
        st["sizer"].params = params
        return st
    if kind == "batch":
        st["tables"] = tables = _mix_tables(case, seed)
        st["queries"] = _mix_queries(case, seed)
        st["ctx"] = Context()
        st["runner"] = B.BatchRunner(tables, "learned", _trained_sizer(), B.PlainRunner(st["ctx"], tables))
        return st
    ctx = st["ctx"] = Context()
    if kind in ("q1", "q6"):
        _register(ctx, {"fact": _fact(case, seed)})
        spec = f"template=q1;ship_le={case['ship_le']}" if kind == "q1" else "template=q6"
    elif kind == "join":
        dim, probe = _dim_probe(case, seed)
        _register(ctx, {"dim": dim, "probe": probe})
        spec = f"template=join_topk;od_lt={case['od_lt']};ship_gt={case['ship_gt']};k={case['k']}"
    elif kind == "multi_join":
        _register(ctx, _snowflake(case, seed))
        spec = "template=multi_join"
    else:
        ranks, key, r = _skewed(case, seed)
        n = case["rows"]
        _register(ctx, {"zprobe": {"z_key": key[ranks], "z_value": r.ints(90_000, 10_500_000, n, torch.int64)}})
        del ranks
        ctx.register_symbol("zgroups", case["keys"])
        if kind == "hashjoin":
            order = r.perm(case["keys"])
            _register(ctx, {"zbuild": {"zb_key": key[order], "zb_payload": r.ints(0, 1_000_000, case["keys"], torch.int32)}})
        if kind == "groups_sorted":
            st["host"] = torch.empty((3, case["keys"]), dtype=torch.int64).pin_memory().numpy()
        spec = {"groupby": "template=groupby", "groups_sorted": "template=groupby_sorted",
                "hashjoin": "template=hashjoin"}[kind]
    torch.cuda.synchronize()
    st["query"] = ctx.prepare(spec)
    return st


def run(state):
    kind = state["kind"]
    if kind == "sizer":
        g, loss = state["sizer"].grads(state["X"], state["Y"])
        return {"grads": g, "loss": float(loss)}
    if kind == "batch":
        return _batch_answer(state["case"], state["queries"], state["runner"].run(state["queries"])[0])
    ctx, q = state["ctx"], state["query"]
    if kind == "groups_sorted":
        ctx.run(q, collect=False)
        n = int(ctx.read_buffer("gss_n", np.uint64, 1)[0])
        h = state["host"]
        return {c: ctx.read_buffer(name, np.int64, n, out=h[i])
                for i, (c, name) in enumerate((("key", "gss_out_k"), ("count", "gss_out_c"), ("sum", "gss_out_v")))}
    if kind in ("groupby", "hashjoin"):
        return ctx.run(q, arrays=True)[0]
    res, _ = ctx.run(q)
    out = {c: res.column(c) for c in res.columns}
    return {c: [ord(x) for x in v] if v and isinstance(v[0], str) else v for c, v in out.items()}


def _batch_answer(case, queries, results):
    """The answers as arrays: (count, sum) per scalar query, the top lists,
    and each group-by's counts and sums indexed by key."""
    scalars, tops, cards = [], [], [q.card for q in queries if q.tmpl == "groupby"]
    counts, sums = np.zeros(sum(cards), np.int64), np.zeros(sum(cards), np.int64)
    off = 0
    for q, r in zip(queries, results):
        if r[0] == "scalar":
            scalars.append((r[1], r[2]))
        elif r[0] == "topk":
            tops.append(list(r[1]) + [(-1, -1)] * (q.k - len(r[1])))
        else:
            k, c, s = (r[1][:, 0], r[1][:, 1], r[1][:, 2]) if r[0] == "groups_raw" else r[1:]
            counts[off + k] = c
            sums[off + k] = s
            off += q.card
    return {"scalars": np.array(scalars, np.int64).reshape(-1, 2), "tops": np.array(tops, np.int64).reshape(-1, 10, 2),
            "group_counts": counts, "group_sums": sums}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    flops = 0
    if kind == "q1":
        nbytes = 38 * case["rows"]
    elif kind == "q6":
        nbytes = 28 * case["rows"]
    elif kind == "join":
        # price and discount only of the matched rows
        share = 0.2 * min(1.0, case["od_lt"] / 2406)
        late = sum(1 for d in range(0, 2406, 6) if d < case["od_lt"] and d + 61 > case["ship_gt"]) / max(
            1, sum(1 for d in range(0, 2406, 6) if d < case["od_lt"]))
        nbytes = 9 * case["dim"] + 8 * case["probe"] + 16 * case["probe"] * share * late
    elif kind in ("groupby", "groups_sorted"):
        nbytes = 16 * case["rows"] + 24 * min(case["keys"], case["rows"])
    elif kind == "hashjoin":
        nbytes = 8 * case["rows"] + 12 * case["keys"] + 24 * case["keys"]
    elif kind == "multi_join":
        # price and discount only of the kept lines: the order's date and region, the same nation
        kept = case["lines"] * (365 / 2406) * (1 / 5) * (1 / 25)
        nbytes = 8 * (case["cust"] + case["supp"] + case["lines"]) + 12 * case["orders"] + 16 * kept
    elif kind == "batch":
        nbytes = 0
        for q in _mix_queries(case, 0):
            nbytes += B.query_bytes(q, MIX_DIM_ROWS)
            if q.tmpl == "groupby":
                nbytes += 24 * min(q.card, q.rows)
    else:
        nbytes = 4 * (18 * case["rows"] + 2 * 9538)
        flops = 6 * 9344 * case["rows"]
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------
# the same answers by plain torch / numpy in 64 bits
# ---------------------------------------------------------------------------
def exact(case, seed):
    kind = case["kind"]
    if kind == "q1":
        return _exact_q1(case, _fact(case, seed))
    if kind == "q6":
        t = _fact(case, seed)
        day, disc = t["f_ship_day"], t["f_discount"]
        m = (day >= 365) & (day < 730) & (disc >= 5) & (disc <= 7) & (t["f_quantity"] < 24)
        return {"revenue": [int((t["f_price"] * disc)[m].sum())]}
    if kind == "join":
        dim, probe = _dim_probe(case, seed)
        keep = torch.zeros(case["dim"] + 1, device="cuda", dtype=torch.bool)
        keep[dim["b_key"].long()] = (dim["b_segment"] == 1) & (dim["b_order_day"] < case["od_lt"])
        fk = probe["p_fk"].long()
        m = keep[fk] & (probe["p_ship_day"] > case["ship_gt"])
        rev = (probe["p_price"] * (100 - probe["p_discount"]))[m]
        k, v = _top(fk[m], rev, case["dim"] + 1, case["k"])
        return {"key": k.tolist(), "revenue": v.tolist()}
    if kind in ("groupby", "groups_sorted"):
        ranks, key, r = _skewed(case, seed)
        val = r.ints(90_000, 10_500_000, case["rows"], torch.int64)
        c, s = _per_key(ranks, val, case["keys"])
        at = torch.nonzero(c).flatten()
        k, c, s = key[at], c[at], s[at]
        o = torch.argsort(k)
        if kind == "groups_sorted":
            o = o[torch.argsort(s[o], descending=True, stable=True)]
        return {"key": k[o].cpu().numpy(), "count": c[o].cpu().numpy(), "sum": s[o].cpu().numpy()}
    if kind == "hashjoin":
        ranks, key, r = _skewed(case, seed)
        r.ints(90_000, 10_500_000, case["rows"], torch.int64)
        order = r.perm(case["keys"])
        payload = torch.zeros(case["keys"], device="cuda", dtype=torch.int64)
        payload[order] = r.ints(0, 1_000_000, case["keys"], torch.int32).long()
        c = torch.bincount(ranks, minlength=case["keys"])
        at = torch.nonzero(c).flatten()
        o = at[torch.argsort(key[at])]
        return {"key": key[o].cpu().numpy(), "count": c[o].cpu().numpy(), "sum": (c * payload)[o].cpu().numpy()}
    if kind == "multi_join":
        t = _snowflake(case, seed)
        o, ln = t["ord"], t["line"]
        ok = (o["o_day"] >= 730) & (o["o_day"] < 1095)
        nat = torch.where(ok, t["cust"]["c_nation"][o["o_cust"].long() - 1], -1)
        nat = torch.where(nat % 5 == 2, nat, -1)
        cn, sn = nat[ln["l_okey"].long() - 1], t["supp"]["s_nation"][ln["l_supp"].long() - 1]
        m = (cn >= 0) & (cn == sn)
        rev = torch.zeros(25, device="cuda", dtype=torch.int64)
        rev.index_add_(0, cn[m].long(), (ln["l_price"] * (100 - ln["l_discount"]))[m])
        at = torch.nonzero(rev).flatten()
        return {"nation": at.tolist(), "revenue": rev[at].tolist()}
    if kind == "batch":
        return _exact_batch(case, seed)
    return _exact_sizer(*_sizer_data(case, seed))


def _per_key(keys, values, n):
    c = torch.bincount(keys, minlength=n)
    s = torch.zeros(n, device="cuda", dtype=torch.int64)
    s.index_add_(0, keys, values)
    return c, s


def _top(keys, values, n, k):
    """The k keys of largest sum, ties by key."""
    c, s = _per_key(keys, values, n)
    at = torch.nonzero(c).flatten()
    o = torch.argsort(s[at], descending=True, stable=True)[:k]
    return at[o], s[at][o]


def _exact_q1(case, t):
    a, b = t["f_flag_a"].long(), t["f_flag_b"].long()
    bucket = torch.where(a == ord("A"), 0, torch.where(a == ord("N"), 2, 4)) + (b != ord("F"))
    m = t["f_ship_day"] <= case["ship_le"]
    bucket, qty, price = bucket[m], t["f_quantity"][m], t["f_price"][m]
    disc, tax = t["f_discount"][m], t["f_tax"][m]
    count = torch.bincount(bucket, minlength=6)

    def total(v):
        return torch.zeros(6, device="cuda", dtype=torch.int64).index_add_(0, bucket, v)

    at = torch.nonzero(count).flatten()
    n = count[at].tolist()
    out = {"flag_a": [ord("ANR"[i // 2]) for i in at.tolist()], "flag_b": [ord("FO"[i % 2]) for i in at.tolist()]}
    sums = {"sum_qty": qty, "sum_base_price": price, "sum_disc_price": price * (100 - disc),
            "sum_charge": price * (100 - disc) * (100 + tax), "sum_disc": disc}
    sums = {c: total(v)[at].tolist() for c, v in sums.items()}
    out.update(sums, count_order=n)
    for name, of in (("avg_qty", "sum_qty"), ("avg_price", "sum_base_price"), ("avg_disc", "sum_disc")):
        out[name] = [float(s) / c for s, c in zip(sums[of], n)]
    return out


def _exact_batch(case, seed):
    tables, queries, results = _mix_tables(case, seed), _mix_queries(case, seed), []
    attr = torch.zeros(MIX_DIM_ROWS + 1, device="cuda", dtype=torch.int32)
    attr[tables.dim["md_key"].long()] = tables.dim["md_attr"]
    for q in queries:
        t = {c: v[q.row0:q.row0 + q.rows] for c, v in tables.tables[q.table].items()}
        m = t["m_filter"] < q.thr
        if q.tmpl == "join":
            m &= attr[t["m_fk"].long()] < q.attr_lt
        v = t["m_value"][m]
        if q.tmpl in ("agg", "join"):
            results.append(("scalar", int(v.numel()), int(v.sum())))
            continue
        keys = t[q.key][m].long() % q.card
        if q.tmpl == "topk":
            k, s = _top(keys, v, q.card, q.k)
            results.append(("topk", list(zip(k.tolist(), s.tolist()))))
        else:
            c, s = _per_key(keys, v, q.card)
            results.append(("groups", np.arange(q.card), c.cpu().numpy(), s.cpu().numpy()))
    return _batch_answer(case, queries, results)


def _exact_sizer(params, X, Y):
    """Mean squared error and its gradient at the weights rounded to BF16."""
    p = torch.from_numpy(params).to(torch.bfloat16).double()
    shapes, ws, off = ((64, 16), (64, 64), (64, 64), (2, 64)), [], 0
    for o, i in shapes:
        ws += [p[off:off + o * i].view(o, i), p[off + o * i:off + o * i + o]]
        off += o * i + o
    for w in ws:
        w.requires_grad_(True)
    x, y = torch.from_numpy(X).double(), torch.from_numpy(Y).double()
    h = x
    for j in range(3):
        h = torch.relu(h @ ws[2 * j].T + ws[2 * j + 1])
    loss = ((h @ ws[6].T + ws[7] - y) ** 2).mean()
    g = torch.autograd.grad(loss, ws)
    return {"grads": torch.cat([v.reshape(-1) for v in g]).numpy(), "loss": float(loss)}
