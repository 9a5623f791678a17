"""Performance cases of the hash groupby framework: calls a program makes
through the public API (GroupBy, BatchGroupBy, inner_join), over the sizes,
types and requests of the repository's own workloads.

Groups (and join pairs) come back in no particular order, so every case does
what a program does next: it puts the result rows in key order (a batch's and
a join's into arrays indexed by key or left row).  Those are the case's
outputs.  Inputs are made on the device from the seed.
"""
from __future__ import annotations

import math
import os

import torch

import cudf_b200
from cudf_b200 import (BatchGroupBy, BatchInstance, Column, GroupBy, GroupByRequest, NullPolicy, Table, Tune,
                       TypeId)
from cudf_b200 import aggregation as agg
from cudf_b200.column import storage_dtype
from cudf_b200.join import inner_join

_TUNE_TABLE = os.path.join(os.path.dirname(os.path.abspath(cudf_b200.__file__)), "tuning", "batch_tune.txt")
_QUANTILES = (0.25, 0.5, 0.9)
_TORCH = {"int8": torch.int8, "int16": torch.int16, "int32": torch.int32, "int64": torch.int64,
          "float32": torch.float32, "float64": torch.float64}


def listed():
    return [
        # a served request at the small end: launches and host latency
        {"name": "served_10k", "kind": "served", "rows": 10_007, "groups": 100},
        # a served request of ordinary size
        {"name": "served_1m", "kind": "served", "rows": 1_000_003, "groups": 30_000},
        # the largest served request: high cardinality, one value column
        {"name": "served_50m", "kind": "served", "rows": 50_000_000, "groups": 10_000_000},
        # a data-frame style groupby: int32 key, one double column, no nulls
        {"name": "frame_10m", "kind": "frame", "rows": 10_000_000, "groups": 1_000},
        # the 100M-row workload (two value columns, one with nulls, six
        # aggregations on each) over its four cardinalities
        {"name": "plain_1e2", "kind": "plain", "rows": 100_000_000, "groups": 100},
        {"name": "plain_1e4", "kind": "plain", "rows": 100_000_000, "groups": 10_000},
        {"name": "plain_1e6", "kind": "plain", "rows": 100_000_000, "groups": 1_000_000},
        {"name": "plain_1e8", "kind": "plain", "rows": 100_000_000, "groups": 100_000_000},
        # skewed composite key with null keys
        {"name": "zipf_200m", "kind": "zipf", "rows": 200_000_000, "groups": 100_000},
        # thousands of independent groupbys in one graph launch
        {"name": "batch_4096", "kind": "batch", "instances": 4096, "rows_max": 1_000_000},
        # order statistics (the kinds that sort each group's values)
        {"name": "quantiles_100m", "kind": "quantiles", "rows": 100_000_000, "groups": 10_000},
        # a fact table joined to a dimension table with unique keys
        {"name": "join_50m", "kind": "join", "rows": 50_000_000, "groups": 1_000_000},
    ]


def draw(rng):
    def log_uniform(lo, hi):
        return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))

    kind = rng.choice(["served", "served", "plain", "plain", "plain", "frame", "zipf", "batch", "quantiles", "join"])
    if kind == "served":
        rows = log_uniform(1e4, 5e7)
        return {"kind": kind, "rows": rows, "groups": log_uniform(1e2, min(1e7, rows))}
    if kind == "plain":
        rows = log_uniform(1e5, 1e8)
        return {"kind": kind, "rows": rows, "groups": log_uniform(10, rows)}
    if kind == "frame":
        return {"kind": kind, "rows": log_uniform(1e5, 5e7), "groups": log_uniform(10, 1e5)}
    if kind == "zipf":
        return {"kind": kind, "rows": log_uniform(1e6, 2e8), "groups": log_uniform(1e3, 1e5)}
    if kind == "batch":
        return {"kind": kind, "instances": log_uniform(64, 4096), "rows_max": log_uniform(1e5, 1e6)}
    if kind == "quantiles":
        return {"kind": kind, "rows": log_uniform(1e5, 1e8), "groups": log_uniform(10, 1e5)}
    return {"kind": kind, "rows": log_uniform(1e5, 5e7), "groups": log_uniform(1e3, 5e6)}


# ------------------------------------------------------------------ inputs

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _bits(valid):
    """Bool tensor -> validity bitmask words (int32, LSB-first), 64-byte padded."""
    n = valid.numel()
    v = torch.zeros((n + 511) // 512 * 512, dtype=torch.uint8, device=valid.device)
    v[:n] = valid
    w = torch.tensor([1, 2, 4, 8, 16, 32, 64, 128], dtype=torch.uint8, device=valid.device)
    return (v.view(-1, 8) * w).sum(dim=1, dtype=torch.uint8).view(torch.int32)


def _batch_shape(case):
    """Rows and cardinality of each instance: log-uniform, one fixed list per
    case (a batch is planned for its row counts)."""
    g = torch.Generator()
    g.manual_seed(int(case["instances"]))
    u = torch.rand(case["instances"], 2, generator=g, dtype=torch.float64)
    rows = torch.exp(math.log(1e3) + u[:, 0] * math.log(case["rows_max"] / 1e3)).long()
    cards = torch.exp(math.log(10.0) + u[:, 1] * math.log(1e4 / 10.0)).long()
    return rows, cards


def _inputs(case, seed):
    """The case's raw columns, as torch tensors."""
    g = _generator(seed)
    kind = case["kind"]
    d = {"device": "cuda", "generator": g}
    if kind == "batch":
        rows, cards = _batch_shape(case)
        total = int(rows.sum())
        inst = torch.repeat_interleave(torch.arange(case["instances"], device="cuda"), rows.cuda())
        u = torch.rand(total, dtype=torch.float64, **d)
        k = (u * cards.cuda()[inst]).to(torch.int32)
        return {"k": k, "v": torch.randint(0, 1_000_000_001, (total,), **d), "inst": inst}
    n, c = case["rows"], case["groups"]
    if kind == "served":
        return {"k": torch.randint(0, c, (n,), **d), "v": torch.randn(n, dtype=torch.float64, **d)}
    if kind == "frame":
        return {"k": torch.randint(0, c, (n,), dtype=torch.int32, **d), "v": torch.randn(n, dtype=torch.float64, **d)}
    if kind in ("plain", "quantiles"):
        return {"k": torch.randint(0, c, (n,), **d), "a": torch.randint(-1_000_000, 1_000_001, (n,), **d),
                "b": torch.randn(n, dtype=torch.float32, **d), "bv": torch.rand(n, **d) >= 0.10}
    if kind == "join":
        # unique dimension keys spread over the int64 range; a tenth of the facts match none
        m = c + c // 9
        keys = (torch.randperm(m, **d) + 1) * 982_451_653
        return {"build": keys[:c].clone(), "probe": keys[torch.randint(0, m, (n,), **d)]}
    # zipf: distinct (int32, int16) pairs, rank drawn by inverse CDF with s = 1.2
    pair = torch.unique(torch.randint(-2 ** 47, 2 ** 47, (c + c // 8 + 64,), **d))
    pair = pair[torch.randperm(pair.numel(), **d)][:c]
    cdf = torch.cumsum(torch.arange(1, c + 1, dtype=torch.float64, device="cuda") ** -1.2, 0)
    cdf /= cdf[-1].clone()
    j = torch.empty(n, dtype=torch.int32, device="cuda")
    for lo in range(0, n, 1 << 26):
        hi = min(n, lo + (1 << 26))
        u = torch.rand(hi - lo, dtype=torch.float64, **d)
        j[lo:hi] = torch.searchsorted(cdf, u, right=True).clamp_(max=c - 1)
    v = torch.randn(n, dtype=torch.float64, **d).exp_()
    return {"pair": pair, "rank": j, "v": v, "v1": torch.rand(n, **d) >= 0.02, "v2": torch.rand(n, **d) >= 0.02}


_SIX = (agg.sum, agg.count, agg.min, agg.max, agg.mean, agg.variance)


def prepare(case, seed):
    x = _inputs(case, seed)
    kind = case["kind"]
    if kind == "batch":
        rows, cards = _batch_shape(case)
        first = torch.cumsum(rows, 0) - rows
        insts = []
        for n, s in zip(rows.tolist(), first.tolist()):
            insts.append(BatchInstance(Table([Column(TypeId.INT32, n, x["k"], None, s)]),
                                       [GroupByRequest(Column(TypeId.INT64, n, x["v"], None, s),
                                                       [agg.sum(), agg.count(), agg.max()])]))
        batch = BatchGroupBy(insts, tune=Tune.CACHED, tune_file=_TUNE_TABLE)
        base = (torch.cumsum(cards, 0) - cards).cuda()
        groups = int(cards.sum())
        dense = [torch.zeros(groups, dtype=t, device="cuda") for t in (torch.int64, torch.int32, torch.int64)]
        return {"case": case, "batch": batch, "base": base, "dense": dense}
    n, c = case["rows"], case["groups"]
    i32, i64, f32, f64 = torch.int32, torch.int64, torch.float32, torch.float64
    if kind == "served":
        req = [GroupByRequest(Column(TypeId.FLOAT64, n, x["v"]), [agg.sum(), agg.count(), agg.mean()])]
        return {"case": case, "keys": Table([Column(TypeId.INT64, n, x["k"])]), "req": req,
                "out": _sorted(case, i64, f64, i32, f64)}
    if kind == "frame":
        req = [GroupByRequest(Column(TypeId.FLOAT64, n, x["v"]),
                              [agg.sum(), agg.count(), agg.mean(), agg.min(), agg.max()])]
        return {"case": case, "keys": Table([Column(TypeId.INT32, n, x["k"])]), "req": req,
                "out": _sorted(case, i32, f64, i32, f64, f64, f64)}
    if kind in ("plain", "quantiles"):
        a = Column(TypeId.INT64, n, x["a"])
        b = Column(TypeId.FLOAT32, n, x["b"], _bits(x["bv"]), 0, n - int(x["bv"].sum()))
        keys = Table([Column(TypeId.INT64, n, x["k"])])
        if kind == "plain":
            req = [GroupByRequest(a, [f() for f in _SIX]), GroupByRequest(b, [f() for f in _SIX])]
            out = _sorted(case, i64, i64, i32, i64, i64, f64, f64, f32, i32, f32, f32, f64, f64)
            return {"case": case, "keys": keys, "req": req, "out": out}
        req = [GroupByRequest(a, [agg.median(), agg.quantile(_QUANTILES), agg.nunique()]),
               GroupByRequest(b, [agg.nth_element(0, NullPolicy.INCLUDE), agg.m2()])]
        return {"case": case, "keys": keys, "req": req,
                "out": _sorted(case, i64, f64, (f64, len(_QUANTILES)), i32, f32, f64)}
    if kind == "join":
        return {"case": case, "left": Table([Column(TypeId.INT64, n, x["probe"])]),
                "right": Table([Column(TypeId.INT64, c, x["build"])]),
                "dense": torch.full((n,), -1, dtype=torch.int32, device="cuda")}
    p1, p2 = (x["pair"] >> 16).to(torch.int32), x["pair"].to(torch.int16)
    rank = x["rank"].long()
    k1 = Column(TypeId.INT32, n, p1[rank], _bits(x["v1"]), 0, n - int(x["v1"].sum()))
    k2 = Column(TypeId.INT16, n, p2[rank], _bits(x["v2"]), 0, n - int(x["v2"].sum()))
    req = [GroupByRequest(Column(TypeId.FLOAT64, n, x["v"]), [agg.sum(), agg.mean()])]
    return {"case": case, "keys": Table([k1, k2]), "req": req, "out": _sorted(case, i64, f64, f64)}


# -------------------------------------------------------------------- run

def _data(col):
    """A result column's elements as a tensor (a view of its buffer)."""
    dt = storage_dtype(col.type_id)
    return col.data[:col.size * dt.itemsize].view(_TORCH[dt.name])


def _sorted(case, *dtypes):
    """Result arrays with room for every key: the keys, then one per result column."""
    rows = min(case["rows"], case["groups"])
    return [torch.zeros(rows, dtype=t, device="cuda") if not isinstance(t, tuple)
            else torch.zeros(rows, t[1], dtype=t[0], device="cuda") for t in dtypes]


def _by_key(out, key, cols):
    """The keys in ascending order, and the result columns in that order, into the arrays `out`."""
    n = key.numel()
    key, order = torch.sort(key)
    out[0][:n] = key
    for o, c in zip(out[1:], cols):
        torch.index_select(c, 0, order, out=o[:n])
    return out + [n]


def run(state):
    kind = state["case"]["kind"]
    if kind == "batch":
        r = state["batch"].execute()
        groups = torch.from_numpy(r.offsets[1:] - r.offsets[:-1]).cuda()
        at = torch.repeat_interleave(state["base"], groups, output_size=r.num_groups) + _data(r.keys[0])
        return [d.index_copy_(0, at, _data(c)) for d, c in zip(state["dense"], r.results[0].columns())]
    if kind == "join":
        left, right = inner_join(state["left"], state["right"])
        state["dense"].index_copy_(0, _data(left).long(), _data(right))
        return [state["dense"], left.size]
    keys, res = GroupBy(state["keys"]).aggregate(state["req"])
    cols = [c for t in res for c in t.columns()]
    nulls = [c.null_count for c in cols]
    cols = [_data(c) for c in cols]
    if kind == "zipf":
        pair = (_data(keys[0]).long() << 16) | (_data(keys[1]).long() & 0xffff)
        return _by_key(state["out"], pair, cols) + nulls
    if kind == "quantiles":
        cols[1] = cols[1].view(-1, len(_QUANTILES))
    return _by_key(state["out"], _data(keys[0]), cols) + nulls


# ------------------------------------------------------------------- exact

def _sums(k, x, c):
    return torch.zeros(c, dtype=x.dtype, device=x.device).index_add_(0, k, x)


def _extreme(k, x, c, how):
    out = torch.zeros(c, dtype=x.dtype, device=x.device)
    return out.scatter_reduce_(0, k, x, how, include_self=False)


def _moments(k, x, c):
    """Rows, sum, mean and centred sum of squares per key, in double."""
    n = _sums(k, torch.ones_like(k), c)
    s = _sums(k, x, c)
    mean = torch.where(n > 0, s / n, torch.zeros_like(s))
    return n, s, mean, _sums(k, (x - mean[k]).square_(), c)


def _variance(n, m2):
    return torch.where(n > 1, m2 / (n - 1).clamp(min=1), torch.zeros_like(m2))


def _rows(case, g, cols):
    """The rows of the groups `g` as _by_key lays them out."""
    rows = min(case["rows"], case["groups"])
    out = []
    for c in cols:
        p = torch.zeros((rows,) + tuple(c.shape[1:]), dtype=c.dtype, device=c.device)
        p[:g.numel()] = c
        out.append(p)
    return out + [g.numel()]


def exact(case, seed):
    x = _inputs(case, seed)
    kind = case["kind"]
    if kind == "batch":
        rows, cards = _batch_shape(case)
        at = (torch.cumsum(cards, 0) - cards).cuda()[x["inst"]] + x["k"]
        c = int(cards.sum())
        return [_sums(at, x["v"], c), _sums(at, torch.ones_like(at), c), _extreme(at, x["v"], c, "amax")]
    n, c = case["rows"], case["groups"]
    if kind == "join":
        order = torch.argsort(x["build"])
        sorted_build = x["build"][order]
        at = torch.searchsorted(sorted_build, x["probe"]).clamp_(max=c - 1)
        hit = sorted_build[at] == x["probe"]
        return [torch.where(hit, order[at], torch.full_like(at, -1)).to(torch.int32), int(hit.sum())]
    if kind == "zipf":
        pairs, order = torch.sort(x["pair"])
        place = torch.empty(c, dtype=torch.int64, device="cuda")
        place[order] = torch.arange(c, device="cuda")
        keep = x["v1"] & x["v2"]
        cnt, s, mean, _ = _moments(place[x["rank"][keep].long()], x["v"][keep], c)
        g = torch.nonzero(cnt)[:, 0]
        return _rows(case, g, [pairs[g], s[g], mean[g]]) + [0, 0]
    k = x["k"].long()
    if kind in ("served", "frame"):
        cnt, s, mean, _ = _moments(k, x["v"], c)
        out = [s, cnt, mean]
        if kind == "frame":
            out += [_extreme(k, x["v"], c, "amin"), _extreme(k, x["v"], c, "amax")]
        g = torch.nonzero(cnt)[:, 0]
        return _rows(case, g, [g] + [o[g] for o in out]) + [0] * len(out)
    a, b, bv = x["a"], x["b"].double(), x["bv"]
    kb, xb = k[bv], b[bv]
    nb, sb, mb, m2b = _moments(kb, xb, c)
    if kind == "plain":
        na, _, ma, m2a = _moments(k, a.double(), c)
        g = torch.nonzero(na)[:, 0]
        out = [_sums(k, a, c), na, _extreme(k, a, c, "amin"), _extreme(k, a, c, "amax"), ma, _variance(na, m2a),
               sb, nb, _extreme(kb, xb, c, "amin"), _extreme(kb, xb, c, "amax"), mb, _variance(nb, m2b)]
        empty = int((nb[g] == 0).sum())
        nulls = [0, 0, 0, 0, 0, int((na == 1).sum()), empty, 0, empty, empty, empty, int((nb[g] < 2).sum())]
        return _rows(case, g, [g] + [o[g] for o in out]) + nulls
    val, i = torch.sort(a)
    key, i = torch.sort(k[i], stable=True)
    val = val[i]
    cnt = torch.bincount(key, minlength=c)
    start = torch.cumsum(cnt, 0) - cnt
    new = torch.ones_like(key)
    new[1:] = (key[1:] != key[:-1]) | (val[1:] != val[:-1])
    uniq = _sums(key, new, c)
    row = _extreme(k, torch.arange(n, device="cuda"), c, "amin")
    first = torch.where(bv[row], b[row], torch.zeros_like(b[row]))
    g = torch.nonzero(cnt)[:, 0]
    cnt, start = cnt[g], start[g]

    def quantile(p):
        pos = (cnt - 1).double() * p
        lo = pos.floor().long()
        hi = torch.minimum(lo + 1, cnt - 1)
        x0, x1 = val[start + lo].double(), val[start + hi].double()
        return x0 + (pos - lo) * (x1 - x0)

    nulls = [0, 0, 0, int((~bv[row][g]).sum()), int((nb[g] == 0).sum())]
    quantiles = torch.stack([quantile(p) for p in _QUANTILES], 1)
    return _rows(case, g, [g, quantile(0.5), quantiles, uniq[g], first[g], m2b[g]]) + nulls


# -------------------------------------------------------- work, tolerance

def _distinct(rows, groups):
    """Expected distinct keys among `rows` uniform draws from `groups`."""
    return groups * -math.expm1(-rows / groups)


def work(case):
    """Each input read once and each result row written once; one operation per accumulator and row."""
    kind = case["kind"]
    if kind == "batch":
        rows, cards = _batch_shape(case)
        g = sum(_distinct(n, c) for n, c in zip(rows.tolist(), cards.tolist()))
        return {"bytes": int(rows.sum()) * 12 + g * 24, "flops": int(rows.sum()) * 3}
    n, c = case["rows"], case["groups"]
    if kind == "join":
        return {"bytes": 8 * n + 8 * c + 0.9 * n * 8, "flops": n}
    g = _distinct(n, c)
    row, out, ops = {"served": (16, 28, 2), "frame": (12, 40, 4), "plain": (20.125, 85.75, 14),
                     "zipf": (14.25, 22, 2), "quantiles": (20.125, 60, 30)}[kind]
    return {"bytes": n * row + g * out, "flops": n * ops}


def tolerance(case):
    """Sums are taken in 64 bits, so results differ only by the order of the
    additions (and a float32 SUM by its last rounding)."""
    kind = case["kind"]
    if kind in ("batch", "join"):
        return "exact"
    return {"rel": 1e-10, "max": 5e-7}
