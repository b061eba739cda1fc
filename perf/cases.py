"""The calls whose speed this library is judged by, over the sizes they are used at.

A case is a dict of plain values.  `listed()` gives the fixed ones, `draw(rng)` one more of the
same ranges; `prepare` makes what a program holds before the call (device columns made from the
seed, a validated segmentation, a captured pipeline), `run` is one pass through the public entry
points, `work` the bytes a pass cannot do without, and `exact` the same results from plain torch
in 64 bits.

Length-changing calls leave their count on the device; `run` reads it, as a program does that goes
on with the rows, and returns exactly those rows.  u32 columns are handed over as int32 views
(torch indexes and compares those everywhere).
"""
import math

import torch

import massively_b200 as mb
from massively_b200 import lazy, op, pipeline, seg, vector

SIGN = -(1 << 31)
_executors = {}


def _exec():
    """One executor for the process, as a program keeps one per device."""
    if "ex" not in _executors:
        _executors["ex"] = mb.Executor(0)
    return _executors["ex"]


# ------------------------------------------------------------------ cases --

def listed():
    return [
        # The headline: a stable sort of (u32 key, u32 value) pairs, keys uniform over 32 bits.
        {"name": "sort_pairs_u32_2e28", "kind": "sort_pairs", "n": 1 << 28, "key": "u32",
         "key_bits": 32},
        # The same call as a small request of a serving loop: launches and latency.
        {"name": "sort_pairs_u32_small", "kind": "sort_pairs", "n": 3001, "key": "u32",
         "key_bits": 32},
        # 64-bit keys alone (ids, timestamps), an ordinary ragged size.
        {"name": "sort_keys_u64", "kind": "sort_keys", "n": (1 << 22) - 3, "key": "u64"},
        # Prefix sums of the largest column the benchmark uses.
        {"name": "scan_u32_2e30", "kind": "scan", "n": 1 << 30, "type": "u32", "inclusive": True},
        # Float prefix sums, a ragged large size: the deterministic fold.
        {"name": "scan_f32_large", "kind": "scan", "n": (1 << 28) + 3, "type": "f32",
         "inclusive": True},
        # Prefix sums of a small request (offsets of a batch of lengths).
        {"name": "scan_u32_small", "kind": "scan", "n": 1500, "type": "u32", "inclusive": False},
        # A filter with its predicate fused onto the column, half of the rows kept.
        {"name": "copy_where_u32", "kind": "copy_where", "n": (1 << 28) - 3, "columns": 1},
        # filter -> sort -> aggregate -> join over Zipf keys, captured once and replayed.
        {"name": "group_by_2e27", "kind": "group_by", "n": 1 << 27, "distinct": 1 << 20,
         "kept": 0.3},
        # Two sorted columns of unequal ragged lengths into one.
        {"name": "merge_u32", "kind": "merge", "left": 100000007, "right": 150000001},
        # The join's multiset intersection of two sorted lists with duplicates.
        {"name": "set_intersection_u32", "kind": "set_intersection", "left": (1 << 25) - 39,
         "right": 30000001},
        # Per-segment prefix sums: many uneven segments (lognormal lengths) in one call.
        {"name": "seg_scan_f32_2e26", "kind": "seg_scan", "n": 1 << 26, "segments": 1 << 20},
        # Per-segment sorts of the same shape.
        {"name": "seg_sort_u32_2e26", "kind": "seg_sort", "n": 1 << 26, "segments": 1 << 20},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sort_pairs", "sort_keys", "scan", "copy_where", "group_by", "merge",
                       "set_intersection", "seg_scan", "seg_sort"])
    if kind == "sort_pairs":
        return {"kind": kind, "n": _log(rng, 1 << 10, 1 << 28),
                "key": rng.choice(["u32", "u32", "i32", "f32"]),
                "key_bits": rng.choice([32, 32, 16])}
    if kind == "sort_keys":
        return {"kind": kind, "n": _log(rng, 1 << 12, 1 << 26), "key": rng.choice(["u64", "i64"])}
    if kind == "scan":
        return {"kind": kind, "n": _log(rng, 1 << 10, 1 << 29),
                "type": rng.choice(["u32", "f32", "i64"]), "inclusive": rng.random() < 0.5}
    if kind == "copy_where":
        return {"kind": kind, "n": _log(rng, 1 << 10, 1 << 27), "columns": rng.choice([1, 2])}
    if kind == "group_by":
        n = _log(rng, 1 << 16, 1 << 26)
        return {"kind": kind, "n": n, "distinct": _log(rng, 1 << 10, min(1 << 20, n // 4)),
                "kept": round(rng.uniform(0.1, 0.9), 3)}
    if kind in ("merge", "set_intersection"):
        top = 1 << (27 if kind == "merge" else 24)
        return {"kind": kind, "left": _log(rng, 1 << 10, top), "right": _log(rng, 1 << 10, top)}
    n = _log(rng, 1 << 12, 1 << 26)
    return {"kind": kind, "n": n, "segments": max(1, int(n / _log(rng, 16, 512)))}


# ----------------------------------------------------------------- inputs --

def _bits32(g, n):
    """Uniform 32-bit words, as int32."""
    return torch.randint(SIGN, 1 << 31, (n,), generator=g, device="cuda", dtype=torch.int32)


def _u32(ex, t):
    return ex.from_tensor(t.view(torch.uint32))


def _draws(g, n, span):
    """n numbers drawn uniformly from [0, span)."""
    return torch.randint(0, span, (n,), generator=g, device="cuda", dtype=torch.int64)


def _sorted_u32(x):
    """Numbers below 2^32 as a sorted u32 list (int32 bits)."""
    return torch.sort(x).values.to(torch.int32)


def _shared(case):
    """The items a set_intersection case's lists have in common."""
    return min(case["left"], case["right"]) // 2


def _offsets(g, n, segments):
    """Segment offsets with lognormal(3, 1.5) lengths scaled to sum to n (empty ones among them)."""
    z = torch.randn(segments, generator=g, device="cuda", dtype=torch.float64)
    ends = torch.cumsum(torch.exp(3.0 + 1.5 * z), 0)
    off = torch.zeros(segments + 1, device="cuda", dtype=torch.int64)
    off[1:] = torch.floor(ends / ends[-1] * n).to(torch.int64).clamp_(max=n)
    off[-1] = n
    return off


def _flags(g, n, kept):
    """u32 flags, `kept` of n set, in random places."""
    return (torch.randperm(n, generator=g, device="cuda") < kept).to(torch.int32)


def _spread(rank):
    """The key of a rank: ranks spread over the 32-bit space by a bijection."""
    return (rank * 2654435761 & 0xFFFFFFFF).to(torch.int32)


def _rows(case, g):
    """Group-by rows: u32 Zipf(1.1) keys spread over 32 bits, f32 N(0, 1) values, u32 flags.
    Every key has one kept row at least, so the number of groups is the same for every seed."""
    n, distinct = case["n"], case["distinct"]
    w = torch.arange(1, distinct + 1, device="cuda", dtype=torch.float64) ** -1.1
    cdf = torch.cumsum(w, 0)
    u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * cdf[-1]
    rank = torch.searchsorted(cdf, u, right=True).clamp_(max=distinct - 1)
    del u
    step = n // distinct
    once = torch.arange(distinct, device="cuda") * step + \
        torch.randint(0, step, (distinct,), generator=g, device="cuda")
    rank[once] = torch.randperm(distinct, generator=g, device="cuda")
    keys = _spread(rank)
    values = torch.randn(n, generator=g, device="cuda", dtype=torch.float32)
    flags = (torch.rand(n, generator=g, device="cuda") < case["kept"]).to(torch.int32)
    flags[once] = 1
    return keys, values, flags


def _unsigned(t):
    """int32 bits of u32 values as int64 numbers."""
    return t.to(torch.int64) & 0xFFFFFFFF


def _inputs(case, seed):
    """The plain torch tensors of a case: from the seed alone."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    kind = case["kind"]
    if kind == "sort_pairs":
        n = case["n"]
        if case["key"] == "f32":
            k = torch.randn(n, generator=g, device="cuda", dtype=torch.float32)
        elif case["key_bits"] == 16:
            k = torch.randint(0, 1 << 16, (n,), generator=g, device="cuda", dtype=torch.int32)
        else:
            k = _bits32(g, n)
        return k, torch.arange(n, device="cuda", dtype=torch.int32)
    if kind == "sort_keys":
        n = case["n"]
        hi = torch.randint(SIGN, 1 << 31, (n,), generator=g, device="cuda", dtype=torch.int64)
        lo = torch.randint(0, 1 << 32, (n,), generator=g, device="cuda", dtype=torch.int64)
        return ((hi << 32) | lo,)
    if kind == "scan":
        if case["type"] == "f32":
            return (torch.randn(case["n"], generator=g, device="cuda", dtype=torch.float32),)
        if case["type"] == "i64":
            return (torch.randint(-1000000, 1000000, (case["n"],), generator=g, device="cuda",
                                  dtype=torch.int64),)
        return (_bits32(g, case["n"]),)
    if kind == "copy_where":
        cols = [_bits32(g, case["n"]) for _ in range(case["columns"])]
        flags = _flags(g, case["n"], case["n"] // 2)
        if case["columns"] == 1:  # the predicate is IsEven of the column: bit 0 is the flag's
            return (cols[0] & -2 | (1 - flags),)
        return tuple(cols) + (flags,)
    if kind == "group_by":
        # a sorted list, half of it keys of the rows
        d = case["distinct"]
        other = torch.cat([torch.randperm(d, generator=g, device="cuda")[:d // 2],
                           d + torch.arange(d - d // 2, device="cuda")])
        other = torch.sort(_unsigned(_spread(other))).values.to(torch.int32)
        return _rows(case, g) + (other,)
    if kind == "merge":
        return tuple(_sorted_u32(_draws(g, case[k], 1 << 32)) for k in ("left", "right"))
    if kind == "set_intersection":
        # values x * 3 with the copies both lists hold (half of the shorter one), x * 3 + 1 in the
        # left list alone and x * 3 + 2 in the right alone; each with duplicates
        span = max(case["left"], case["right"])
        both = _draws(g, _shared(case), span) * 3
        return tuple(_sorted_u32(torch.cat([both, _draws(g, case[k] - both.numel(), span) * 3 + j]))
                     for j, k in ((1, "left"), (2, "right")))
    off = _offsets(g, case["n"], case["segments"])
    if kind == "seg_scan":
        return torch.randn(case["n"], generator=g, device="cuda", dtype=torch.float32), off
    return _bits32(g, case["n"]), off


def prepare(case, seed):
    ex = _exec()
    kind = case["kind"]
    x = _inputs(case, seed)
    st = {"case": case, "ex": ex}
    if kind == "sort_pairs":
        k = x[0].view(torch.uint32) if case["key"] == "u32" else x[0]
        st["keys"], st["values"] = ex.from_tensor(k), _u32(ex, x[1])
    elif kind == "sort_keys":
        st["keys"] = ex.from_tensor(x[0].view(torch.uint64) if case["key"] == "u64" else x[0])
    elif kind == "scan":
        st["x"] = ex.from_tensor(x[0].view(torch.uint32) if case["type"] == "u32" else x[0])
    elif kind == "copy_where":
        st["cols"] = [_u32(ex, t) for t in x]
    elif kind == "group_by":
        keys, values, flags, other = x
        cols = (_u32(ex, keys), ex.from_tensor(values), _u32(ex, flags), _u32(ex, other))
        st["rows"] = cols
        st["captured"] = pipeline.Captured(ex, lambda e: pipeline.group_by(e, *cols))
    elif kind in ("merge", "set_intersection"):
        st["left"], st["right"] = _u32(ex, x[0]), _u32(ex, x[1])
    else:
        values = ex.from_tensor(x[0] if kind == "seg_scan" else x[0].view(torch.uint32))
        sg = seg.Segmentation.from_offsets(ex, _u32(ex, x[1].to(torch.int32)))
        st["segments"] = sg.segments(values)
    return st


# -------------------------------------------------------------------- run --

def _plain(v):
    t = v.tensor
    if t.dtype == torch.uint32:
        return t.view(torch.int32)
    return t.view(torch.int64) if t.dtype == torch.uint64 else t


def run(state):
    case, ex = state["case"], state["ex"]
    kind = case["kind"]
    if kind == "sort_pairs":
        k, v = vector.radix_sort_pairs(ex, state["keys"], state["values"])
        return [_plain(k), _plain(v)]
    if kind == "sort_keys":
        return [_plain(vector.sort(ex, state["keys"]))]
    if kind == "scan":
        if case["inclusive"]:
            return [_plain(vector.inclusive_scan(ex, state["x"], op.Add))]
        return [_plain(vector.exclusive_scan(ex, state["x"], 7, op.Add))]
    if kind == "copy_where":
        cols = state["cols"]
        if case["columns"] == 1:
            kept = vector.copy_where(ex, cols[0], lazy.map(cols[0], op.IsEven))
            return [_plain(kept)[:kept.logical_len()]]
        kept = vector.copy_where(ex, mb.zip2(cols[0], cols[1]), cols[2])
        n = kept.cols[0].logical_len()
        return [_plain(c)[:n] for c in kept.cols]
    if kind == "group_by":
        cap = state["captured"]
        cap.replay()
        out = cap.outputs
        n, m = out["keys"].logical_len(), out["common"].logical_len()
        return [_plain(out[k])[:n] for k in ("keys", "sum", "count", "min")] + \
            [_plain(out["common"])[:m]]
    if kind == "merge":
        return [_plain(vector.merge(ex, state["left"], state["right"]))]
    if kind == "set_intersection":
        common = vector.set_intersection(ex, state["left"], state["right"])
        return [_plain(common)[:common.logical_len()]]
    how = seg.InclusiveScan(op.Add) if kind == "seg_scan" else seg.Sort()
    return [_plain(seg.ForEachSegment(how).run(ex, state["segments"]).values())]


def work(case):
    """Every input read once and every output written once."""
    kind = case["kind"]
    if kind == "sort_pairs":
        return {"bytes": 16 * case["n"], "flops": 0}
    if kind == "sort_keys":
        return {"bytes": 16 * case["n"], "flops": 0}
    if kind == "scan":
        return {"bytes": (16 if case["type"] == "i64" else 8) * case["n"], "flops": 0}
    if kind == "copy_where":
        return {"bytes": (6 if case["columns"] == 1 else 16) * case["n"], "flops": 0}
    if kind == "group_by":
        return {"bytes": 12 * case["n"] + 22 * case["distinct"], "flops": 0}
    if kind == "merge":
        return {"bytes": 8 * (case["left"] + case["right"]), "flops": 0}
    if kind == "set_intersection":
        return {"bytes": 4 * (case["left"] + case["right"] + _shared(case)), "flops": 0}
    return {"bytes": 8 * case["n"] + 4 * (case["segments"] + 1), "flops": 0}


# ------------------------------------------------------------------ exact --

def exact(case, seed):
    kind = case["kind"]
    x = _inputs(case, seed)
    if kind == "sort_pairs":
        k, v = x
        order = torch.sort(k ^ SIGN if case["key"] == "u32" else k, stable=True).indices
        return [k[order], v[order]]
    if kind == "sort_keys":
        if case["key"] == "i64":
            return [torch.sort(x[0]).values]
        flip = -(1 << 63)
        return [torch.sort(x[0] ^ flip).values ^ flip]
    if kind == "scan":
        if case["type"] == "f32":
            s = torch.cumsum(x[0], 0, dtype=torch.float64)
            return [s if case["inclusive"] else 7 + torch.cat([s.new_zeros(1), s[:-1]])]
        s = torch.cumsum(x[0], 0, dtype=torch.int64)
        if not case["inclusive"]:
            s = 7 + torch.cat([s.new_zeros(1), s[:-1]])
        return [s if case["type"] == "i64" else s.to(torch.int32)]
    if kind == "copy_where":
        if case["columns"] == 1:
            return [x[0][(x[0] & 1) == 0]]
        return [c[x[2] != 0] for c in x[:2]]
    if kind == "group_by":
        keys, values, flags, other = x
        keep = flags != 0
        k, where, count = torch.unique(_unsigned(keys[keep]), return_inverse=True,
                                       return_counts=True)
        v = values[keep].to(torch.float64)
        total = torch.zeros(k.numel(), device="cuda", dtype=torch.float64).index_add_(0, where, v)
        least = torch.full((k.numel(),), math.inf, device="cuda", dtype=torch.float64)
        least.scatter_reduce_(0, where, v, "amin")
        common = k[torch.isin(k, _unsigned(other))]
        return [k.to(torch.int32), total, count.to(torch.int32), least, common.to(torch.int32)]
    if kind == "merge":
        return [torch.sort(torch.cat([_unsigned(t) for t in x])).values.to(torch.int32)]
    if kind == "set_intersection":
        left, right = x
        first = torch.searchsorted(left, left)
        copy = torch.arange(left.numel(), device="cuda") - first
        have = torch.searchsorted(right, left, right=True) - torch.searchsorted(right, left)
        return [left[copy < have]]
    values, off = x
    ids = torch.searchsorted(off, torch.arange(case["n"], device="cuda"), right=True) - 1
    if kind == "seg_sort":
        key = (ids << 32) | _unsigned(values)
        return [torch.sort(key).values.to(torch.int32)]
    # Sums restart at each segment: the running sum (in integers of 2^-36, which every f32 above
    # 2^-13 in size is a multiple of)
    # less its value before the segment's first item.
    scaled = torch.round(values.to(torch.float64) * float(1 << 36)).to(torch.int64)
    run_sum = torch.cumsum(scaled, 0)
    before = torch.cat([run_sum.new_zeros(1), run_sum])[off[ids]]
    return [(run_sum - before).to(torch.float64) / float(1 << 36)]
