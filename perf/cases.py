"""Performance cases of the framework: what a user of it has it do, through the public Engine API.

Each case is a dict with a "kind" (which operator) and its sizes and options:

  groupby   hash GROUP BY over device-resident columns (Engine.execute_groupby)
  batch     many small GROUP BY queries over one resident table (Engine.execute_batch)
  pairs     INNER join index pairs (Engine.hash_join_indices)
  joinagg   fused JOIN -> GROUP BY (Engine.join_groupby)
  sort      ORDER BY permutation over one or two keys (Engine.sort_indices)
  compact   WHERE compaction of a whole table (Engine.compact_columns)

Sizes come from bench.py's workloads, the h2o.ai db-benchmark shapes the reference publishes (10M rows;
100 groups, 10K groups, 1M groups) and the repository's tests. Inputs are made on the GPU from the seed:
the keys' values, the row order and the value columns follow it, while which rows share a group (or match, or
pass a filter) is fixed by the case up to that order, so the outputs of two seeds have the same shapes.
"""

from __future__ import annotations

import functools
import importlib
import math

import numpy as np
import torch

bolt = importlib.import_module("craton-bolt_b200")

DEV = "cuda:0"
GIB = 1 << 30


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # A dashboard query over a small table: host work, launches and latency are all of it. The row count is
        # odd and no hint is given, as when the caller knows nothing of the table.
        {"name": "groupby_20k", "kind": "groupby", "rows": 20_011, "groups": 100, "keys": "i32", "aggs": "sum_i64",
         "skew": 0.0, "where": 0, "nulls": 0, "hint": False},
        # The plain single-key GROUP BY of the benchmark: 1M rows, 1,024 groups.
        {"name": "groupby_1m", "kind": "groupby", "rows": 1_000_000, "groups": 1024, "keys": "i32",
         "aggs": "sum_i64", "skew": 0.0, "where": 0, "nulls": 0, "hint": True},
        # h2o q4: AVG over three float columns, 10M rows, 100 groups.
        {"name": "groupby_avg3_10m", "kind": "groupby", "rows": 10_000_000, "groups": 100, "keys": "i32",
         "aggs": "avg3_f64", "skew": 0.0, "where": 0, "nulls": 0, "hint": True},
        # h2o q5's shape with a nullable value column: 10M rows over 1M groups without skew (more groups than
        # any on-chip table holds), 5 % NULLs.
        {"name": "groupby_nulls_10m", "kind": "groupby", "rows": 10_000_000, "groups": 1_000_000, "keys": "i64",
         "aggs": "sum_f64", "skew": 0.0, "where": 0, "nulls": 5, "hint": True},
        # The benchmark's headline: filtered two-key GROUP BY, 100M rows, Zipf pairs, every aggregate.
        {"name": "groupby_filtered_100m", "kind": "groupby", "rows": 100_000_000, "groups": 10_000_000,
         "keys": "i32x2", "aggs": "full", "skew": 1.1, "where": 50, "nulls": 0, "hint": True},
        # Keys that do not pack into 64 bits (Int64 x Int32): 10M rows, 1M groups.
        {"name": "groupby_wide_10m", "kind": "groupby", "rows": 10_000_000, "groups": 1_000_000, "keys": "i64x32",
         "aggs": "wide", "skew": 0.0, "where": 0, "nulls": 0, "hint": True},
        # A dashboard's refresh: 32 filtered queries over 10K to 1M rows of one resident table, as one batch.
        {"name": "batch_32", "kind": "batch", "queries": 32, "rows_min": 10_000, "rows_max": 1_000_000,
         "groups": 1000, "skew": 1.1, "where": 50},
        # A dimension table joined to a fact table, the pairs wanted: 1M x 20M rows, 90 % of the probes match.
        {"name": "pairs_1m_20m", "kind": "pairs", "build": 1_000_000, "probe": 20_000_000, "match": 90,
         "dup": 1},
        # The benchmark's join -> GROUP BY: 10M build rows, 200M probe rows, Decimal128 amounts, 100 groups.
        {"name": "joinagg_10m_200m", "kind": "joinagg", "build": 10_000_000, "probe": 200_000_000, "match": 90,
         "groups": 100},
        # ORDER BY category DESC (nullable, few values), price: 10M rows, two keys.
        {"name": "sort_2key_10m", "kind": "sort", "rows": 10_000_000, "keys": "i32n,f32", "range": 1000},
        # The benchmark's ORDER BY: 268M int64 keys over the full range.
        {"name": "sort_i64_268m", "kind": "sort", "rows": 1 << 28, "keys": "i64", "range": 0},
        # The benchmark's WHERE compaction: 100M rows, five columns and the row ids.
        {"name": "compact_100m", "kind": "compact", "rows": 100_000_000, "keep": 50, "mask": False, "nulls": 0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["groupby", "groupby", "groupby", "batch", "pairs", "joinagg", "sort", "sort", "compact"])
    if kind == "groupby":
        keys = rng.choice(["i32", "i32", "i64", "i32x2", "i32x2", "i64x32"])
        aggs = "wide" if keys == "i64x32" else rng.choice(["sum_i64", "count", "sum_f64", "avg3_f64", "full"])
        rows = _log(rng, 5_000, 20_000_000 if keys == "i64x32" else 80_000_000)
        groups = _log(rng, 1_000 if keys == "i64x32" else 10, max(2_000, min(rows // 2, 4_000_000)))
        return {"kind": kind, "rows": rows, "groups": groups, "keys": keys, "aggs": aggs,
                "skew": rng.choice([0.0, 1.1]), "where": 0 if keys == "i64x32" else rng.choice([0, 10, 50, 90]),
                "nulls": rng.choice([0, 0, 5]), "hint": rng.random() < 0.75}
    if kind == "batch":
        return {"kind": kind, "queries": _log(rng, 8, 32), "rows_min": _log(rng, 5_000, 20_000),
                "rows_max": _log(rng, 50_000, 1_000_000), "groups": _log(rng, 50, 20_000),
                "skew": rng.choice([0.0, 1.1]), "where": rng.choice([0, 50])}
    if kind == "pairs":
        return {"kind": kind, "build": _log(rng, 1_000, 10_000_000), "probe": _log(rng, 10_000, 40_000_000),
                "match": rng.choice([10, 50, 90, 100]), "dup": rng.choice([1, 1, 2])}
    if kind == "joinagg":
        return {"kind": kind, "build": _log(rng, 1_000, 10_000_000), "probe": _log(rng, 10_000, 150_000_000),
                "match": rng.choice([50, 90, 100]), "groups": _log(rng, 4, 20_000)}
    if kind == "sort":
        keys = rng.choice(["i64", "f32", "f64", "i32", "i64n", "i32n,f32", "i32,i64"])
        return {"kind": kind, "rows": _log(rng, 5_000, 60_000_000 if "," in keys else 150_000_000), "keys": keys,
                "range": rng.choice([0, _log(rng, 10, 1 << 30)])}
    return {"kind": kind, "rows": _log(rng, 10_000, 90_000_000), "keep": rng.choice([1, 10, 50, 90]),
            "mask": rng.random() < 0.3, "nulls": rng.choice([0, 0, 5])}


# ---------------------------------------------------------------------------
# Inputs (torch on the GPU, from the seed alone)
# ---------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _turn(x, seed):
    """The rows in another order for every seed."""
    return torch.roll(x, (int(seed) * 2654435761) % max(1, x.shape[0]))


def _mix(x):
    """A bijection of int64 (murmur3's finaliser), so distinct ranks stay distinct keys."""
    def lsr(v, k):
        return (v >> k) & ((1 << (64 - k)) - 1)
    x = x ^ lsr(x, 33)
    x = x * -49064778989728563
    x = x ^ lsr(x, 33)
    x = x * -4265267296055464877
    return x ^ lsr(x, 33)


def _key_base(seed):
    return (int(seed) % 4096) << 40


@functools.lru_cache(maxsize=4)
def _zipf_p(groups, skew):
    w = np.arange(1, groups + 1, dtype=np.float64) ** (-skew)
    return w / w.sum()


def _ranks(g, n, groups, skew):
    """Group ranks in [0, groups): uniform, or Zipf(skew) through the inverse CDF."""
    if not skew:
        return torch.randint(0, groups, (n,), generator=g, device=DEV, dtype=torch.int64)
    c = torch.from_numpy(np.cumsum(_zipf_p(groups, skew))).to(DEV)  # (on the host: the same bits every time)
    out = torch.empty(n, dtype=torch.int64, device=DEV)
    for s in range(0, n, 1 << 25):
        m = min(1 << 25, n - s)
        u = torch.rand(m, generator=g, device=DEV, dtype=torch.float64)
        out[s:s + m] = torch.searchsorted(c, u, right=True).clamp_(max=groups - 1)
    return out


def _validity(g, n, pct):
    """Arrow validity bitmap with about `pct` percent NULLs."""
    m = (n + 7) // 8
    keep = torch.rand(m * 8, generator=g, device=DEV) >= pct / 100.0
    w = torch.tensor([1, 2, 4, 8, 16, 32, 64, 128], dtype=torch.int32, device=DEV)
    return (keep.view(m, 8).to(torch.int32) * w).sum(1).to(torch.uint8)


def _valid_mask(v, n):
    b = torch.tensor([0, 1, 2, 3, 4, 5, 6, 7], dtype=torch.uint8, device=DEV)
    return ((v.view(-1, 1) >> b) & 1).view(-1)[:n].bool()


def _f64(g, n, sigma=1e3):
    return torch.randn(n, generator=g, device=DEV, dtype=torch.float64) * sigma


def _i32(g, n, hi):
    return torch.randint(0, hi, (n,), generator=g, device=DEV, dtype=torch.int32)


def _full_i64(g, n):
    return torch.randint(-(1 << 63), (1 << 63) - 1, (n,), generator=g, device=DEV, dtype=torch.int64)


def _groupby_inputs(c, seed, turn=True):
    """(table, key names, aggregates, where) of a groupby case."""
    g, fixed = _gen(seed), _gen(0)
    n, keys = c["rows"], c["keys"]
    rank = _ranks(fixed, n, c["groups"], c["skew"])
    rank = _turn(rank, seed) if turn else rank
    t = {}
    if keys == "i32":
        t["k"] = bolt.col((rank + int(seed) % 100_000).to(torch.int32))
    elif keys == "i64":
        t["k"] = bolt.col(_mix(rank + _key_base(seed)))
    elif keys == "i32x2":
        h = _mix(rank + _key_base(seed))
        t["a"] = bolt.col((h >> 32).to(torch.int32))
        t["b"] = bolt.col(h.to(torch.int32))
        del h
    else:  # an account number and a day
        t["a"] = bolt.col(_mix((rank >> 4) + _key_base(seed)))
        t["b"] = bolt.col((rank & 15).to(torch.int32))
    del rank
    names = list(t)
    where = []
    if c["where"]:
        f = _i32(fixed, n, 100)
        t["f"] = bolt.col(_turn(f, seed) if turn else f)
        where = [("f", "<", c["where"])]
    aggs = []
    if c["aggs"] in ("sum_i64", "wide"):
        t["v"] = bolt.col(torch.randint(-1_000_000, 1_000_001, (n,), generator=g, device=DEV, dtype=torch.int64))
        aggs = [("sum", "v"), ("count_star", None)] if c["aggs"] == "wide" else [("sum", "v")]
    if c["aggs"] in ("sum_f64", "wide", "full", "batch"):
        t["x"] = bolt.col(_f64(g, n))
        aggs += {"batch": [("sum", "x")], "sum_f64": [("sum", "x"), ("count_star", None)], "wide": [("avg", "x")],
                 "full": [("sum", "x"), ("avg", "x"), ("count_star", None)]}[c["aggs"]]
    if c["aggs"] == "count":
        aggs = [("count_star", None)]
    if c["aggs"] == "avg3_f64":
        for v in ("x", "y", "z"):
            t[v] = bolt.col(_f64(g, n, 100.0))
            aggs.append(("avg", v))
    if c["aggs"] == "full":
        t["i"] = bolt.col(_full_i64(g, n))
        aggs += [("min", "i"), ("max", "i")]
    if c["nulls"]:
        for name in t:
            if name in ("v", "x"):
                t[name].validity = _validity(g, n, c["nulls"])
    return t, names, aggs, where


def _expected_groups(n, groups, skew):
    """Expected distinct groups among n rows."""
    if n <= 0:
        return 0
    if not skew:
        return int(round(groups * -math.expm1(n * math.log1p(-1.0 / groups)))) if groups > 1 else 1
    return int(round(float(-np.expm1(n * np.log1p(-_zipf_p(groups, skew))).sum())))


def _batch_table(c):
    return {"rows": 2 * c["rows_max"], "groups": c["groups"], "keys": "i32", "aggs": "batch", "skew": c["skew"],
            "where": c["where"], "nulls": 0}


def _batch_spans(c):
    """Row spans of the batch's queries over the resident table (log-uniform lengths)."""
    r = np.random.default_rng(5)
    n = np.exp(r.uniform(np.log(c["rows_min"]), np.log(c["rows_max"]), c["queries"])).astype(np.int64)
    begin = (r.random(c["queries"]) * (2 * c["rows_max"] - n)).astype(np.int64)
    return [(int(b), int(b + m)) for b, m in zip(begin, n)]


def _join_keys(c, seed):
    """Build keys (each occurring `dup` times, shuffled) and probe keys of which `match` percent occur."""
    g, fixed = _gen(seed), _gen(0)
    npr, dup = c["probe"], c.get("dup", 1)
    distinct = max(1, c["build"] // dup)
    nb = distinct * dup
    off = _key_base(seed)
    bk = _mix(torch.arange(nb, device=DEV, dtype=torch.int64) % distinct + off)
    if dup > 1:
        bk = bk[torch.randperm(nb, generator=g, device=DEV)]
    pk = torch.empty(npr, dtype=torch.int64, device=DEV)
    for s in range(0, npr, 1 << 26):
        m = min(1 << 26, npr - s)
        idx = torch.randint(0, distinct, (m,), generator=g, device=DEV, dtype=torch.int64)
        hit = _turn(torch.rand(m, generator=fixed, device=DEV) * 100.0 < c["match"], seed)
        pk[s:s + m] = _mix(torch.where(hit, idx, idx + distinct) + off)
    return g, bk, pk


def _sort_column(g, n, spec, rng_):
    """One ORDER BY key column; `rng_` values when given (0: the type's whole range)."""
    ty, null = spec.rstrip("n"), spec.endswith("n")
    if ty in ("i32", "i64"):
        lo, hi = (0, rng_) if rng_ else ((-(1 << 31), (1 << 31) - 1) if ty == "i32" else (-(1 << 63), (1 << 63) - 1))
        v = torch.randint(lo, hi, (n,), generator=g, device=DEV, dtype=torch.int32 if ty == "i32" else torch.int64)
    else:
        dt = torch.float32 if ty == "f32" else torch.float64
        # Prices and measurements over many magnitudes, both signs; a few zeros, infinities and NaNs.
        v = torch.pow(10.0, torch.rand(n, generator=g, device=DEV, dtype=dt) * 60 - 30)
        v *= torch.randint(0, 2, (n,), generator=g, device=DEV).to(dt) * 2 - 1
        sel = torch.rand(n, generator=g, device=DEV)
        v[sel < 0.001] = 0.0
        v[(sel >= 0.001) & (sel < 0.002)] = -0.0
        v[(sel >= 0.002) & (sel < 0.003)] = float("inf")
        v[(sel >= 0.003) & (sel < 0.004)] = float("nan")
    return bolt.Column(v, ty, _validity(g, n, 5) if null else None)


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def _scratch(c):
    """Scratch arena of the case's engine."""
    k = c["kind"]
    if k == "sort":
        return c["rows"] * 48 + GIB // 4
    if k == "groupby":
        return max(c["rows"] * 80 + GIB // 4, GIB) if c["keys"] == "i64x32" else 6 * GIB
    if k == "compact":
        return GIB // 2
    if k == "batch":
        return 2 * GIB
    return c["build"] * 160 + c["probe"] // 100 + GIB


def prepare(case, seed):
    c, k = case, case["kind"]
    st = {"case": c}
    if k == "groupby":
        st["table"], st["keys"], st["aggs"], st["where"] = _groupby_inputs(c, seed)
        frac = (c["where"] or 100) / 100.0
        st["hint"] = _expected_groups(int(c["rows"] * frac), c["groups"], c["skew"]) if c["hint"] else 0
    elif k == "batch":
        st["table"], keys, aggs, where = _groupby_inputs(_batch_table(c), seed, turn=False)
    elif k == "pairs":
        _, bk, pk = _join_keys(c, seed)
        st["bk"], st["pk"] = bolt.col(bk), bolt.col(pk)
    elif k == "joinagg":
        g, bk, pk = _join_keys(c, seed)
        amount = torch.zeros((c["probe"], 2), dtype=torch.int64, device=DEV)
        amount[:, 0] = torch.randint(0, 10_000_000, (c["probe"],), generator=g, device=DEV, dtype=torch.int64)
        st["bk"], st["pk"] = bolt.col(bk), bolt.col(pk)
        st["bg"] = bolt.col(_i32(g, c["build"], c["groups"]))
        st["amount"] = bolt.Column(amount, "dec128", None, 2)
    elif k == "sort":
        g = _gen(seed)
        specs = c["keys"].split(",")
        # With two keys the range belongs to the first (the category).
        st["keys"] = [_sort_column(g, c["rows"], s, c["range"] if i == 0 else 0) for i, s in enumerate(specs)]
        st["desc"] = [True, False][:len(specs)] if len(specs) > 1 else [False]
    else:
        t, _, _, _ = _groupby_inputs({"rows": c["rows"], "groups": 10_000_000, "keys": "i32x2", "aggs": "full",
                                      "skew": 0.0, "where": 50, "nulls": c["nulls"]}, seed)
        st["table"], st["where"], st["mask"] = t, [("f", "<", c["keep"])], None
        if c["mask"]:
            st["mask"] = (t["f"].data < c["keep"]).to(torch.uint8)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    st["eng"] = bolt.Engine(0, scratch_bytes=_scratch(c))
    if k == "batch":
        st["queries"] = [st["eng"].prepare_groupby(st["table"], keys, aggs, where=where,
                                                   groups_hint=min(c["groups"], b[1] - b[0]), rows=b,
                                                   out_cap=min(c["groups"], b[1] - b[0]) + 1)
                         for b in _batch_spans(c)]
    return st


def _cols(cs):
    return [[x.data] + ([x.validity] if x.validity is not None else []) for x in cs]


def run(state):
    c, eng = state["case"], state["eng"]
    k = c["kind"]
    if k == "groupby":
        r = eng.execute_groupby(state["table"], state["keys"], state["aggs"], where=state["where"],
                                groups_hint=state["hint"])
        return {"keys": _cols(r.keys), "aggs": _cols(r.aggs)}
    if k == "batch":
        return [{"keys": _cols(r.keys), "aggs": _cols(r.aggs)} for r in eng.execute_batch(state["queries"])]
    if k == "pairs":
        return list(eng.hash_join_indices(state["bk"], state["pk"]))
    if k == "joinagg":
        return _cols(eng.join_groupby(state["bk"], state["bg"], state["pk"], state["amount"],
                                      max_groups=c["groups"] + 1))
    if k == "sort":
        return eng.sort_indices(state["keys"], descending=state["desc"])
    cols, rid = eng.compact_columns(state["table"], where=() if c["mask"] else state["where"], mask=state["mask"])
    return {"cols": _cols(cols.values()), "row_ids": rid}


# ---------------------------------------------------------------------------
# What a pass cannot do without, and how exact its outputs are
# ---------------------------------------------------------------------------
_KEY_BYTES = {"i32": 4, "i64": 8, "i32x2": 8, "i64x32": 12}
_VAL_BYTES = {"sum_i64": 8, "count": 0, "sum_f64": 8, "avg3_f64": 24, "full": 16, "wide": 16}
_OUT_BYTES = {"sum_i64": 8, "count": 8, "sum_f64": 16, "avg3_f64": 24, "full": 40, "wide": 24}


def work(case):
    c, k = case, case["kind"]
    flops = 0
    if k == "groupby":
        frac = (c["where"] or 100) / 100.0
        groups = _expected_groups(int(c["rows"] * frac), c["groups"], c["skew"])
        kb = _KEY_BYTES[c["keys"]]
        row = kb + _VAL_BYTES[c["aggs"]] + (4 if c["where"] else 0)
        by = c["rows"] * row + groups * (kb + _OUT_BYTES[c["aggs"]])
    elif k == "batch":
        rows = sum(e - b for b, e in _batch_spans(c))
        by = rows * (12 + (4 if c["where"] else 0)) + c["queries"] * c["groups"] * 12
    elif k == "pairs":
        by = c["build"] * 8 + c["probe"] * 8 + c["probe"] * c["match"] // 100 * c["dup"] * 8
    elif k == "joinagg":
        by = c["build"] * 12 + c["probe"] * 24 + c["groups"] * 28
    elif k == "sort":
        by = c["rows"] * (sum(int(s[1:3]) // 8 for s in c["keys"].split(",")) + 4)
    else:
        by = c["rows"] * (28 + (1 if c["mask"] else 0)) + c["rows"] * c["keep"] // 100 * 32
    return {"bytes": int(by), "flops": flops}


def _float_aggs(case):
    k = case["kind"]
    return k == "batch" or (k == "groupby" and case["aggs"] not in ("sum_i64", "count"))


def tolerance(case):
    # Whole numbers, keys, permutations and copied values are exact; SUM and AVG over float64 are sums in
    # another order at the same precision (measured against float64 sums in index order: up to 2.7e-14).
    return {"rel": 2e-13} if _float_aggs(case) else "exact"


def _exact_groupby(t, names, aggs, where, rows=None):
    """Float SUM / AVG of every group in float64, in the output's group order; None elsewhere."""
    sl = slice(*rows) if rows else slice(None)
    keep = None
    if where:
        keep = t["f"].data[sl] < where[0][2]

    def take(x):
        return x[sl][keep] if keep is not None else x[sl]
    ks = [take(t[k].data) for k in names]
    if len(ks) == 1:
        packed = ks[0].to(torch.int64)
    elif ks[0].dtype == torch.int32:
        packed = (ks[0].to(torch.int64) << 32) | (ks[1].to(torch.int64) & 0xFFFFFFFF)
    else:  # Int64 x Int32: rank of the first key, then the second
        packed = (torch.unique(ks[0], return_inverse=True)[1] << 32) + ks[1].to(torch.int64)
    u, inv = torch.unique(packed, return_inverse=True)
    out = []
    for op, name in aggs:
        col = t[name] if name else None
        if op not in ("sum", "avg") or col.dtype != "f64":
            out.append([None] * (2 if col is not None and col.validity is not None and op != "count" else 1))
            continue
        v = take(col.data)
        ok = take(_valid_mask(col.validity, col.data.shape[0])) if col.validity is not None else None
        if ok is not None:
            v = torch.where(ok, v, torch.zeros_like(v))
        s = torch.zeros(u.shape[0], dtype=torch.float64, device=DEV).index_add_(0, inv, v)
        if op == "avg":
            one = ok.to(torch.float64) if ok is not None else torch.ones_like(v)
            cnt = torch.zeros_like(s).index_add_(0, inv, one)
            s = torch.where(cnt > 0, s / cnt.clamp(min=1), torch.zeros_like(s))
        out.append([s] + ([None] if ok is not None else []))
    return {"keys": [[None]] * len(names), "aggs": out}


def exact(case, seed):
    if not _float_aggs(case):
        return None
    if case["kind"] == "groupby":
        return _exact_groupby(*_groupby_inputs(case, seed))
    t, names, aggs, where = _groupby_inputs(_batch_table(case), seed, turn=False)
    return [_exact_groupby(t, names, aggs, where, rows=b) for b in _batch_spans(case)]
