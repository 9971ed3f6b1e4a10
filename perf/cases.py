"""The calls whose speed is followed: joins, group-bys, scans with ORDER BY, star batches and served queries.

Every case is one query (or one batch) as a program on top of proteus_gb300 runs it: device columns in hand, one
context with its pool kept for the program's life, results in a defined order.  Where the library leaves the order of
its output open (groups, join pairs), the query has the ORDER BY that a program adds, and the library sorts.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from proteus_gb300 import abi, engine, serve, star

DEV = "cuda"
POOL_BYTES = 40 << 30
COUNT = (abi.AGG_COUNT, abi.VAL_ONE)
AGGS = {
    "product": [COUNT, (abi.AGG_SUM, abi.VAL_PRODUCT)],  # COUNT(*), SUM(R.payload * S.payload)
    "xor": [COUNT, (abi.AGG_SUM, abi.VAL_ROWID_XOR)],  # COUNT(*) and a checksum of the matched row ids
    "mixed": [COUNT, (abi.AGG_SUM, abi.VAL_BUILD), (abi.AGG_MIN, abi.VAL_PROBE), (abi.AGG_MAX, abi.VAL_BUILD)],
}
_context = None


def context():
    """The program's one context."""
    global _context
    if _context is None:
        _context = engine.Context(0, pool_bytes=POOL_BYTES)
    return _context


def listed():
    return [
        # a lookup into a small dimension: launches and host calls are what it costs
        {"name": "join_small", "kind": "join", "build": 4000, "probe": 60_001, "dense": True, "bits": 32, "match": 1.0,
         "copies": 1, "aggs": "product"},
        # the plain join of the benchmark: a 2^20-row dimension with dense surrogate keys, every fact row matches
        {"name": "join_dimension", "kind": "join", "build": 1 << 20, "probe": 1 << 24, "dense": True, "bits": 32,
         "match": 1.0, "copies": 1, "aggs": "product"},
        # int64 keys without a pattern, two build rows a key, a third of the probes without a match, four aggregates
        {"name": "join_int64", "kind": "join", "build": 1_500_000, "probe": 20_000_003, "dense": False, "bits": 64,
         "match": 0.67, "copies": 2, "aggs": "mixed"},
        # scan -> filter -> join -> late materialisation -> ORDER BY: a tenth of 2^24 fact rows, a 2^18-row dimension
        {"name": "filter_join_sort", "kind": "pipeline", "build": 1 << 18, "rows": (1 << 24) + 13, "keep": 0.1,
         "match": 0.8},
        # a partitioned join of ordinary size, payloads on both sides, four aggregates, keys without a pattern
        {"name": "radix_join_medium", "kind": "radix", "build": 3_000_017, "probe": 24_000_001, "dense": False,
         "match": 0.5, "theta": 0.0, "aggs": "mixed"},
        # the large partitioned join of the benchmark: half the probes hit, hits are Zipf
        {"name": "radix_join_large", "kind": "radix", "build": 1 << 27, "probe": 1 << 29, "dense": True, "match": 0.5,
         "theta": 0.5, "aggs": "xor"},
        # GROUP BY a category: few groups, the largest input
        {"name": "groupby_few", "kind": "groupby", "rows": 1 << 29, "groups": 16, "theta": 0.0},
        # GROUP BY a skewed attribute of ordinary size, a row count that is no multiple of anything
        {"name": "groupby_skewed", "kind": "groupby", "rows": 200_000_011, "groups": 1 << 16, "theta": 1.0},
        # GROUP BY a customer key: as many groups as the benchmark has at most
        {"name": "groupby_many", "kind": "groupby", "rows": 1 << 28, "groups": 1 << 24, "theta": 0.0},
        # RadixNest: int64 keys and values
        {"name": "nest_int64", "kind": "nest", "rows": 1 << 27, "groups": 1 << 16},
        # 64 star queries that share one fact scan
        {"name": "star_batch", "kind": "star", "rows": 1 << 28, "queries": 64},
        # a burst of served join + group-by queries of the serving mix
        {"name": "serve_burst", "kind": "serve", "queries": 24, "log_build": 24, "log_probe": 27},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["join", "join", "pipeline", "radix", "radix", "groupby", "groupby", "groupby", "nest", "star",
                       "serve"])
    if kind == "join":
        build = size(1000, 1 << 22)
        return {"kind": kind, "build": build, "probe": size(max(build, 10_000), 1 << 26), "dense": rng.random() < 0.5,
                "bits": rng.choice([32, 32, 64]), "match": round(rng.uniform(0.3, 1.0), 2),
                "copies": rng.choice([1, 1, 2, 3]), "aggs": rng.choice(["product", "xor", "mixed"])}
    if kind == "pipeline":
        return {"kind": kind, "build": size(1000, 1 << 21), "rows": size(1 << 16, 1 << 26),
                "keep": round(rng.uniform(0.02, 0.3), 3), "match": round(rng.uniform(0.3, 1.0), 2)}
    if kind == "radix":
        build = size(1 << 18, 1 << 27)
        return {"kind": kind, "build": build, "probe": size(build, min(1 << 29, 64 * build)),
                "dense": rng.random() < 0.5, "match": round(rng.uniform(0.3, 1.0), 2),
                "theta": rng.choice([0.0, 0.5, 1.0]), "aggs": rng.choice(["xor", "mixed"])}
    if kind == "groupby":
        groups = size(16, 1 << 24)
        return {"kind": kind, "rows": size(max(1 << 14, 4 * groups), 1 << 28), "groups": groups,
                "theta": rng.choice([0.0, 1.0])}
    if kind == "nest":
        groups = size(16, 1 << 22)
        return {"kind": kind, "rows": size(max(1 << 16, 8 * groups), 1 << 27), "groups": groups}
    if kind == "star":
        return {"kind": kind, "rows": size(1 << 18, 1 << 28), "queries": rng.randint(1, 64)}
    return {"kind": kind, "queries": rng.randint(4, 24), "log_build": rng.randint(14, 24),
            "log_probe": rng.randint(18, 27)}


# ------------------------------------------------------------------ inputs
def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _ints(g, n, lo, hi, dtype=torch.int32):
    return torch.randint(lo, hi, (n,), generator=g, device=DEV, dtype=dtype)


def _mix(x, shifts, factors, bits):
    mask = (1 << bits) - 1
    for shift, factor in zip(shifts, factors + (0,)):
        x = x ^ ((x >> shift) & (mask >> shift))
        if factor:
            x = x * factor & mask if bits < 64 else x * factor
    return x


def _spread(x, bits, offset=0):
    """Distinct keys without a pattern for distinct x >= 0: a bijection of the integers of `bits` bits."""
    x = x.long() + offset
    if bits == 64:
        return _mix(x, (30, 27, 31), (0x3F58476D1CE4E5B9, 0x14D049BB133111EB), 64)
    return _mix(x, (16, 15, 15), (0x21F0AAAD, 0x735A2D97), 32).to(torch.int32)  # the low 32 bits, as int32


def _ranks(g, n, count, theta):
    """n ranks in [0, count): uniform, or Zipf-like with exponent theta (the continuous law, rounded down)."""
    if theta == 0.0:
        return _ints(g, n, 0, count)
    out = torch.empty(n, dtype=torch.int32, device=DEV)
    for lo in range(0, n, 1 << 26):
        u = torch.rand(min(1 << 26, n - lo), generator=g, device=DEV, dtype=torch.float64)
        if theta == 1.0:
            r = torch.exp(u * math.log(count + 1.0))
        else:
            r = (u * ((count + 1.0) ** (1.0 - theta) - 1.0) + 1.0) ** (1.0 / (1.0 - theta))
        out[lo:lo + len(u)] = (r - 1.0).clamp_(0, count - 1).to(torch.int32)
    return out


def _keys_of(ids, dense, bits, n):
    """Join keys of ids in [0, 2n): 1..2n, or spread over all values of the type."""
    if dense:
        return (ids + 1).to(torch.int64 if bits == 64 else torch.int32)
    return _spread(ids, bits, 1)


def _join_inputs(case, seed):
    """(build keys, build payload, probe keys, probe payload): `copies` build rows a key; a probe without a match has
    a key of the same law that no build row has."""
    g = _generator(seed)
    nb, np_, bits = case["build"], case["probe"], case.get("bits", 32)
    distinct = max(1, nb // case.get("copies", 1))
    order = torch.randperm(nb, generator=g, device=DEV)
    ids = (order % distinct).to(torch.int32)
    bk = _keys_of(ids, case["dense"], bits, nb)
    pk = torch.empty(np_, dtype=bk.dtype, device=DEV)
    # a Zipf rank's key is that of a build row, which is in random order
    hit = _ranks(g, np_, nb, case.get("theta", 0.0))
    for lo in range(0, np_, 1 << 26):
        r = hit[lo:lo + (1 << 26)].long()
        k = bk[r]
        if case["match"] < 1.0:
            miss = _keys_of(_ints(g, len(r), nb, 2 * nb), case["dense"], bits, nb)
            k = torch.where(torch.rand(len(r), generator=g, device=DEV) < case["match"], k, miss)
        pk[lo:lo + len(r)] = k
    need = case["aggs"] != "xor"
    return bk, _ints(g, nb, 0, 1000) if need else None, pk, _ints(g, np_, 0, 1000) if need else None


def _group_inputs(case, seed):
    """(keys, values, all keys): group keys spread over the type; every group has a row."""
    g = _generator(seed)
    wide = case["kind"] == "nest"
    bits = 64 if wide else 32
    every = _spread(torch.randperm(case["groups"], generator=g, device=DEV), bits, 1 + seed % 1000)
    rank = _ranks(g, case["rows"], case["groups"], case.get("theta", 0.0))
    rank[:case["groups"]] = torch.arange(case["groups"], dtype=torch.int32, device=DEV)
    keys = torch.empty(case["rows"], dtype=every.dtype, device=DEV)
    for lo in range(0, len(keys), 1 << 26):
        keys[lo:lo + (1 << 26)] = every[rank[lo:lo + (1 << 26)].long()]
    del rank
    values = _ints(g, case["rows"], -(1 << 20), 1 << 20, torch.int64 if wide else torch.int32)
    return keys, values, every


def _pipeline_inputs(case, seed):
    """The fact's date, foreign key and price, the dimension's key and attribute, and the range of dates: `keep` of
    the rows are in it, and `match` of those have their foreign key in the dimension."""
    g = _generator(seed)
    n, nb, days = case["rows"], case["build"], 2557
    width = max(1, int(days * case["keep"]))
    first = int(_ints(g, 1, 0, days - width + 1).item())
    order = torch.randperm(n, generator=g, device=DEV)
    kept, matched = int(n * case["keep"]), int(int(n * case["keep"]) * case["match"])
    day = (_ints(g, n, 0, days - width) + (first + width)) % days
    day[order[:kept]] = _ints(g, kept, first, first + width)
    fk = _ints(g, n, 1, 2 * nb + 1)
    fk[order[:matched]] = _ints(g, matched, 1, nb + 1)
    fk[order[matched:kept]] = _ints(g, kept - matched, nb + 1, 2 * nb + 1)
    del order
    key = (torch.randperm(nb, generator=g, device=DEV) + 1).to(torch.int32)
    return day, fk, _ints(g, n, 900, 110_001), key, _ints(g, nb, 0, 250), first, first + width - 1


def _star_inputs(case, seed):
    """Dimensions and queries of the seeded star schema; the fact columns are made on the device."""
    g = _generator(seed)
    dims = star.gen_dims(seed, star.FULL_DIM_ROWS)
    n = case["rows"]
    fk = []
    for dim in dims:
        k = _ints(g, n, 1, dim.n + 1)
        if dim.keys is not None:
            table = torch.from_numpy(dim.keys).to(DEV)
            for lo in range(0, n, 1 << 26):
                k[lo:lo + (1 << 26)] = table[k[lo:lo + (1 << 26)].long() - 1]
        fk.append(k)
    return dims, fk, _ints(g, n, 1, 51), _ints(g, n, 900, 110_001), star.gen_queries(seed, case["queries"], dims)


def _serve_inputs(case, seed):
    """[(build keys, build groups, probe keys, probe values, groups)] of the serving mix.  The sizes are the seeded
    mix's (they are part of the case), the data are the seed's: as many probes match as the match rate says, and they
    go round the build rows, so that as many groups come out for every seed."""
    g = _generator(seed)
    out = []
    for s in serve.gen_shapes(case["queries"], case["queries"], (10, case["log_build"]), (14, case["log_probe"])):
        bk = (torch.randperm(s.n_build, generator=g, device=DEV) + 1).to(torch.int32)
        bg = _spread(torch.arange(s.n_build, device=DEV) % s.cardinality, 32, seed % 1000)
        order = torch.randperm(s.n_probe, generator=g, device=DEV)
        hits = int(s.n_probe * s.match_rate)
        pk = _ints(g, s.n_probe, s.n_build + 1, 1 << 30)
        pk[order[:hits]] = bk[torch.arange(hits, device=DEV) % s.n_build]
        out.append((bk, bg, pk, _ints(g, s.n_probe, 0, 1000), s.cardinality))
    return out


def prepare(case, seed):
    ctx = context()
    kind = case["kind"]
    if kind in ("join", "radix"):
        state = {"cols": _join_inputs(case, seed), "aggs": AGGS[case["aggs"]]}
    elif kind in ("groupby", "nest"):
        keys, values, _ = _group_inputs(case, seed)
        state = {"keys": keys, "values": values}
    elif kind == "pipeline":
        state = {"cols": _pipeline_inputs(case, seed)}
    elif kind == "star":
        dims, fk, qty, price, queries = _star_inputs(case, seed)
        plan = star.StarPlan(ctx, star.StarData(dims, fk, qty, price), fact_tensors=(fk, qty, price))
        out = plan.new_output(len(queries), group_cap=star.GROUPABLE_MAX ** 2)
        for column in ("a", "b", "count", "sum"):
            out[column].zero_()  # rows behind a query's groups are not written
        state = {"plan": plan, "queries": queries, "out": out}
    else:
        server = serve.Server(ctx, hbm_budget=12 << 30, max_batch=64, max_inflight=4, large_slots=2,
                              small_rows=1 << 22)
        queries = [q + (serve.Output(q[4]),) for q in _serve_inputs(case, seed)]
        state = {"server": server, "queries": queries}
    state.update(ctx=ctx, case=case)
    torch.cuda.synchronize()
    return state


# -------------------------------------------------------------------- runs
def _ordered(ctx, keys, *columns):
    """ORDER BY an int32 key: the library sorts (key, row), the other columns follow."""
    rows = torch.arange(len(keys), dtype=torch.int32, device=DEV)
    keys, rows = ctx.sort_by_key([keys, rows], 0)
    return (keys, *(c[rows] for c in columns))


def run(state):
    ctx, case = state["ctx"], state["case"]
    kind = case["kind"]
    if kind == "join":
        bk, bp, pk, pp = state["cols"]
        table = ctx.join_build(bk, bp)
        out = ctx.join_probe_agg(table, pk, pp, state["aggs"])
        table.destroy()
        return out
    if kind == "radix":
        bk, bp, pk, pp = state["cols"]
        return ctx.radix_join_agg(bk, bp, pk, pp, state["aggs"])
    if kind == "groupby":
        cap = min(case["groups"], case["rows"])
        k, c, s, lo, hi, n = ctx.groupby(state["keys"], state["values"], cap, expected_groups=case["groups"])
        n = int(n)
        return _ordered(ctx, k[:n], c[:n], s[:n], lo[:n], hi[:n])
    if kind == "nest":
        cap = min(case["groups"], case["rows"])
        k, c, s, lo, hi, n = ctx.nest_i64(state["keys"], state["values"], cap, expected_groups=case["groups"])
        n = int(n)
        k, order = torch.sort(k[:n])  # the library sorts int32 keys only
        return k, c[order], s[order], lo[order], hi[order]
    if kind == "pipeline":
        day, fk, price, key, attr, first, last = state["cols"]
        rows, n = ctx.select_range(day, first, last)
        rows = rows[:int(n)]
        table = ctx.join_build(key)
        keys = ctx.gather(fk, rows)
        brow, prow, m = ctx.join_probe_pairs(table, keys, len(rows), probe_rows=rows)
        m = int(m)
        table.destroy()
        brow, prow = brow[:m], prow[:m]
        cols = ctx.sort_by_key([prow, ctx.gather(attr, brow), ctx.gather(price, prow)], 0)
        return (*cols, ctx.reduce(cols[2], [COUNT, (abi.AGG_SUM, abi.VAL_BUILD)]))
    if kind == "star":
        out = state["plan"].run(state["queries"], out=state["out"])
        return {k: out[k] for k in ("a", "b", "count", "sum", "n")}
    server = state["server"]
    tickets = server.submit_many(state["queries"])
    for t in tickets:
        if server.wait(t) != abi.OK:
            raise RuntimeError("a served query failed")
    results = []
    for q in state["queries"]:
        o = q[5]
        n = int(o.n)
        results.append(_ordered(ctx, o.group[:n], o.count[:n], o.sum[:n]))
    return [torch.cat([r[j] for r in results]) for j in range(3)]


# ---------------------------------------------------------------- the work
def work(case):
    """Each input column read once, each output written once."""
    kind = case["kind"]
    if kind in ("join", "radix"):
        width = case.get("bits", 32) // 8 + (0 if case["aggs"] == "xor" else 4)
        nbytes = width * (case["build"] + case["probe"]) + 32
    elif kind == "groupby":
        nbytes = 8 * case["rows"] + 28 * case["groups"]
    elif kind == "nest":
        nbytes = 16 * case["rows"] + 40 * case["groups"]
    elif kind == "pipeline":
        kept = case["rows"] * case["keep"]
        nbytes = 4 * case["rows"] + 8 * kept + 8 * case["build"] + 12 * kept * case["match"]
    elif kind == "star":
        nbytes = 24 * case["rows"] + sum(8 * n for n in star.FULL_DIM_ROWS) + 24 * 600 * case["queries"]
    else:
        shapes = serve.gen_shapes(case["queries"], case["queries"], (10, case["log_build"]), (14, case["log_probe"]))
        nbytes = sum(8 * (s.n_build + s.n_probe) + 20 * s.cardinality for s in shapes)
    return {"bytes": nbytes, "flops": 0}


# --------------------------------------------------------------- the values
def _lookup(sorted_keys, keys):
    """(position, found) of keys among distinct sorted keys."""
    at = torch.searchsorted(sorted_keys, keys).clamp_(max=len(sorted_keys) - 1)
    return at, sorted_keys[at] == keys


def _per_key(inverse, n, column):
    """(sum, max) of an int64 column for each of n keys."""
    total = torch.zeros(n, dtype=torch.int64, device=DEV).index_add_(0, inverse, column)
    most = torch.full((n,), -(1 << 62), dtype=torch.int64, device=DEV)
    return total, most.scatter_reduce_(0, inverse, column, "amax")


def _exact_join(case, seed):
    bk, bp, pk, pp = _join_inputs(case, seed)
    keys, inverse = torch.unique(bk, return_inverse=True)
    n = len(keys)
    ones = torch.ones(len(bk), dtype=torch.int64, device=DEV)
    mult = torch.zeros(n, dtype=torch.int64, device=DEV).index_add_(0, inverse, ones)
    kind = case["aggs"]
    first = torch.empty(n, dtype=torch.int64, device=DEV)
    first[inverse] = torch.arange(len(bk), device=DEV)
    copies = int(mult.max())
    rows = [first]  # the build rows of each key, one list for each copy (-1: none)
    left = torch.ones(len(bk), dtype=torch.bool, device=DEV)
    for _ in range(copies - 1):
        left[rows[-1][rows[-1] >= 0]] = False
        idx = torch.nonzero(left).flatten()
        nxt = torch.full((n,), -1, dtype=torch.int64, device=DEV)
        nxt[inverse[idx]] = idx
        rows.append(nxt)
    bsum, bmax = _per_key(inverse, n, bp.long()) if bp is not None else (None, None)
    count = total = 0
    least, most = (1 << 63) - 1, -(1 << 63)
    for lo in range(0, len(pk), 1 << 26):
        at, found = _lookup(keys, pk[lo:lo + (1 << 26)])
        at = at[found]
        count += int(mult[at].sum())
        if kind == "xor":
            prow = torch.nonzero(found).flatten() + lo
            for r in rows:
                b = r[at]
                total += int(torch.where(b >= 0, b ^ prow, 0).sum())
        else:
            pv = pp[lo:lo + (1 << 26)].long()[found]
            total += int((bsum[at] * pv).sum() if kind == "product" else bsum[at].sum())
            if kind == "mixed" and len(at):
                least, most = min(least, int(pv.min())), max(most, int(bmax[at].max()))
    return torch.tensor([count, total] + ([least, most] if kind == "mixed" else []), dtype=torch.int64)


def _exact_groups(keys, values, every):
    every = torch.sort(every)[0]
    n = len(every)
    count, total = (torch.zeros(n, dtype=torch.int64, device=DEV) for _ in range(2))
    least = torch.full((n,), (1 << 63) - 1, dtype=torch.int64, device=DEV)
    most = torch.full((n,), -(1 << 63), dtype=torch.int64, device=DEV)
    for lo in range(0, len(keys), 1 << 26):
        at = torch.searchsorted(every, keys[lo:lo + (1 << 26)])
        v = values[lo:lo + (1 << 26)].long()
        count += torch.bincount(at, minlength=n)
        total.index_add_(0, at, v)
        least.scatter_reduce_(0, at, v, "amin")
        most.scatter_reduce_(0, at, v, "amax")
    some = count > 0
    return tuple(x[some] for x in (every, count, total, least, most))


def exact(case, seed):
    kind = case["kind"]
    if kind in ("join", "radix"):
        return _exact_join(case, seed)
    if kind == "groupby":
        k, c, s, lo, hi = _exact_groups(*_group_inputs(case, seed))
        return k, c, s, lo.to(torch.int32), hi.to(torch.int32)
    if kind == "nest":
        return _exact_groups(*_group_inputs(case, seed))
    if kind == "pipeline":
        day, fk, price, key, attr, first, last = _pipeline_inputs(case, seed)
        order = torch.argsort(key)
        rows = torch.nonzero((day >= first) & (day <= last)).flatten()
        at, found = _lookup(key[order], fk[rows])
        rows = rows[found]
        value = price[rows]
        sums = torch.tensor([len(rows), int(value.long().sum())], dtype=torch.int64)
        return rows.to(torch.int32), attr[order[at[found]]], value, sums
    if kind == "serve":
        parts = []
        for bk, bg, pk, pv, _ in _serve_inputs(case, seed):
            order = torch.argsort(bk)
            groups, inverse = torch.unique(bg, return_inverse=True)
            at, found = _lookup(bk[order], pk)
            at = inverse[order[at[found]]]
            count = torch.bincount(at, minlength=len(groups))
            total = torch.zeros(len(groups), dtype=torch.int64, device=DEV).index_add_(0, at, pv.long()[found])
            some = count > 0
            parts.append((groups[some], count[some], total[some]))
        return [torch.cat([p[j] for p in parts]) for j in range(3)]
    return _exact_star(case, seed)


def _exact_star(case, seed):
    dims, fk, qty, price, queries = _star_inputs(case, seed)
    cap = star.GROUPABLE_MAX ** 2
    out = {k: np.zeros(cap * len(queries), dtype=np.int32 if k in "ab" else np.int64) for k in ("a", "b", "count", "sum")}
    n_groups = np.zeros(len(queries), dtype=np.int64)
    for d, dim in enumerate(dims):  # keys become rows
        if dim.keys is None:
            fk[d] -= 1
        else:
            table = torch.from_numpy(dim.keys).to(DEV)  # ascending
            for lo in range(0, len(qty), 1 << 26):
                fk[d][lo:lo + (1 << 26)] = torch.searchsorted(table, fk[d][lo:lo + (1 << 26)]).to(torch.int32)
    attrs = [[torch.from_numpy(c).to(DEV).long() for c in dim.attrs] for dim in dims]
    for i, q in enumerate(queries):
        joined = [d for d in range(4) if q.join_mask >> d & 1]
        keep = {d: (attrs[d][q.pred_attr[d]] >= q.pred_lo[d]) & (attrs[d][q.pred_attr[d]] <= q.pred_hi[d])
                for d in joined}
        lows = [dims[q.group_dim[k]].lo[q.group_attr[k]] for k in range(2)]
        spans = [dims[q.group_dim[k]].hi[q.group_attr[k]] - lows[k] + 1 for k in range(2)]
        count, total = (torch.zeros(spans[0] * spans[1], dtype=torch.int64, device=DEV) for _ in range(2))
        for lo in range(0, len(qty), 1 << 26):
            rows = None
            for d in joined:
                f = fk[d][lo:lo + (1 << 26)] if rows is None else fk[d][lo + rows]
                ok = torch.nonzero(keep[d][f.long()]).flatten()
                rows = ok if rows is None else rows[ok]
            at = [attrs[q.group_dim[k]][q.group_attr[k]][fk[q.group_dim[k]][lo + rows].long()] - lows[k]
                  for k in range(2)]
            at = at[0] * spans[1] + at[1]
            count += torch.bincount(at, minlength=len(count))
            total.index_add_(0, at, qty[lo + rows].long() * price[lo + rows].long())
        some = torch.nonzero(count).flatten()
        n_groups[i] = m = len(some)
        where = slice(i * cap, i * cap + m)
        out["a"][where] = (some // spans[1] + lows[0]).cpu()
        out["b"][where] = (some % spans[1] + lows[1]).cpu()
        out["count"][where], out["sum"][where] = count[some].cpu(), total[some].cpu()
    return {**out, "n": n_groups}
