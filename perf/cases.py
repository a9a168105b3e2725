"""The GROUP BY work whose time is measured: what one case is, its inputs, one pass through the public operators,
the bytes the pass cannot do without, and the exact result in 64 bits.

Every pass ends as a query does: the aggregates come back ordered (ORDER BY the group keys, or the aggregate where the
keys are strings), so that a result does not depend on the table's slot order.
"""
from __future__ import annotations

import numpy as np
import torch

from qikkdb_b200 import groupby as gb
from qikkdb_b200.batch import GroupByBatch, Query, required_bytes
from qikkdb_b200.groupby import FilterConditions as F

TORCH = {"int32": torch.int32, "int64": torch.int64, "float32": torch.float32, "float64": torch.float64}
NUMPY = {"int32": np.int32, "int64": np.int64, "float32": np.float32, "float64": np.float64}
SIZE = {"int32": 4, "int64": 8, "float32": 4, "float64": 8}
ODD64 = 0x9E3779B97F4A7C15 - (1 << 64)  # odd multipliers: rank -> key is a bijection, so keys spread over the type
ODD32 = 0x9E3779B1


def listed():
    return [
        # One small query as the dispatcher runs it: a new table, one block the size of the sample data set, GetResults.
        # Nothing but launches, allocations and synchronisations.
        dict(name="dispatch_10k", kind="groupby", rows=10_000, keys="int32", spread=False, groups=64, skew=0.0,
             vals="int32", aggs="sum", pred="", keep=1.0, mod=0, fresh=True),
        # The plain known-answer shape at 2^20 rows (8 MB, in L2): every integer aggregate in one table.
        dict(name="plain_1m", kind="groupby", rows=1 << 20, keys="int32", spread=False, groups=1000, skew=0.0,
             vals="int32", aggs="sum,min,max,count", pred="", keep=1.0, mod=0, fresh=False),
        # A few groups over a whole block of trips: GROUP BY passenger_count, AVG and COUNT of a float column.
        dict(name="few_groups_128m", kind="groupby", rows=1 << 27, keys="int32", spread=False, groups=10, skew=1.1,
             vals="float32", aggs="avg,count", pred="", keep=1.0, mod=0, fresh=False),
        # The headline query: WHERE on a float column, skewed 64-bit keys over a million groups.
        dict(name="filtered_256m", kind="groupby", rows=1 << 28, keys="int64", spread=True, groups=1_000_000, skew=1.1,
             vals="float32", aggs="sum,avg", pred="float32", keep=0.5, mod=0, fresh=False),
        # GROUP BY key % m as a served query has it: uniform wide keys, a selective integer WHERE, an odd row count.
        dict(name="modulo_50m", kind="groupby", rows=50_000_017, keys="int64", spread=True, groups=1 << 20, skew=0.0,
             vals="int64", aggs="sum,count,max", pred="int32", keep=0.1, mod=65_521, fresh=False),
        # Two key columns, eight rows to a group: more groups than any on-chip table holds.
        dict(name="composite_128m", kind="composite", rows=1 << 27, side=4096),
        # Columns with NULLs: key and value masks, MIN / MAX / AVG / COUNT of doubles, an odd row count.
        dict(name="nulls_32m", kind="nulls", rows=33_000_001, groups=100_000, vals="float64"),
        # The dispatcher's unfused plan: a filter mask, two compacted columns, then ProcessBlock over them.
        dict(name="compacted_32m", kind="compacted", rows=33_333_333, groups=20_000, keep=0.3),
        # String keys of 8 to 24 bytes, skewed over a million distinct ones, ORDER BY SUM DESC.
        dict(name="strings_32m", kind="strings", rows=1 << 25, groups=1 << 20, longest=24),
        # ORDER BY amount DESC, region ASC over a result of ten million rows, with one column taken in that order.
        dict(name="order_by_10m", kind="order_by", rows=9_999_991, regions=1000),
        # Scalar aggregates under a WHERE.
        dict(name="scalar_256m", kind="scalar", rows=1 << 28, vals="float32", keep=0.5),
        # A dashboard: many small and middling queries in one batch, results on the host.
        dict(name="batch_48", kind="batch", queries=48, least=1000, most=4_000_000),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["groupby"] * 6 + ["composite", "nulls", "compacted", "strings", "order_by", "scalar"])
    if kind == "groupby":
        rows = _log(rng, 5_000, 1 << 27)
        keys = rng.choice(["int32", "int64", "int64", "float32"])
        vals = rng.choice(["int32", "int64", "float32", "float64"])
        mod = _log(rng, 2, 100_000) if keys == "int64" and rng.random() < 0.3 else 0
        return dict(kind=kind, rows=rows, keys=keys, spread=keys != "float32" and rng.random() < 0.6,
                    groups=_log(rng, 4, max(5, min(1_000_000, rows // 4))), skew=rng.choice([0.0, 1.1]), vals=vals,
                    aggs=rng.choice(["sum", "avg,count", "min,max", "sum,min,max,count", "count"]),
                    pred=rng.choice(["", "int32", "float32", "float64"]), keep=round(rng.uniform(0.02, 0.98), 2),
                    mod=mod, fresh=rng.random() < 0.3)
    if kind == "composite":
        rows = _log(rng, 100_000, 1 << 26)
        return dict(kind=kind, rows=rows, side=_log(rng, 8, min(4096, int((rows / 4) ** 0.5))))
    if kind == "nulls":
        rows = _log(rng, 300_000, 33_000_000)
        return dict(kind=kind, rows=rows, groups=_log(rng, 4, max(8, rows // 300)),
                    vals=rng.choice(["int32", "int64", "float32", "float64"]))
    if kind == "compacted":
        rows = _log(rng, 10_000, 33_000_000)
        return dict(kind=kind, rows=rows, groups=_log(rng, 4, min(100_000, rows // 4)),
                    keep=round(rng.uniform(0.02, 0.98), 2))
    if kind == "strings":
        rows = _log(rng, 20_000, 1 << 25)
        return dict(kind=kind, rows=rows, groups=_log(rng, 8, min(1 << 20, rows // 8)), longest=rng.choice([8, 24, 40]))
    if kind == "order_by":
        return dict(kind=kind, rows=_log(rng, 1000, 10_000_000), regions=_log(rng, 2, 100_000))
    return dict(kind=kind, rows=_log(rng, 10_000, 1 << 28), vals=rng.choice(["int32", "int64", "float32", "float64"]),
                keep=round(rng.uniform(0.02, 0.98), 2))


# ---------------------------------------------------------------------------------------------------------------
# Inputs: columns on the GPU, from the seed alone.
# ---------------------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _once(n, groups):
    """One row for every group, evenly through the column: these rows have that group's key and pass every filter, so
    that each group has a result whatever the seed."""
    step = n // groups
    return slice(0, groups * step, step)


def _ranks(g, n, groups, skew):
    """Group numbers in [0, groups): uniform, or Zipf with exponent `skew` (rank 0 the most frequent)."""
    if not skew:
        out = torch.randint(0, groups, (n,), generator=g, device="cuda")
    else:
        cdf = torch.cumsum(torch.arange(1, groups + 1, dtype=torch.float64, device="cuda") ** -skew, 0)
        cdf /= cdf[-1].clone()
        out = torch.empty(n, dtype=torch.int64, device="cuda")
        for a in range(0, n, 1 << 26):
            m = min(1 << 26, n - a)
            u = torch.rand(m, generator=g, dtype=torch.float64, device="cuda")
            out[a:a + m] = torch.searchsorted(cdf, u).clamp_(max=groups - 1)
    out[_once(n, groups)] = torch.randperm(groups, generator=g, device="cuda")
    return out


def _key_of(ranks, dtype, spread):
    """The key that stands for a group number: the number itself, or spread over the whole type."""
    if dtype == "int64":
        return ranks * ODD64 if spread else ranks
    if dtype == "int32":
        return (ranks * ODD32).to(torch.int32) if spread else ranks.to(torch.int32)
    return ranks.to(TORCH[dtype]) * 0.25


def _values(g, n, dtype):
    if dtype == "int32":
        return torch.randint(-1000, 1001, (n,), generator=g, device="cuda", dtype=torch.int32)
    if dtype == "int64":
        return torch.randint(0, 1 << 31, (n,), generator=g, device="cuda")
    return torch.exp(torch.randn(n, generator=g, device="cuda", dtype=TORCH[dtype]) + 2)  # lognormal(2, 1)


def _filter_column(g, n, dtype, keep):
    """A WHERE column and the constant that `col < constant` passes about a share `keep` of the rows with."""
    if dtype in ("int32", "int64"):
        return torch.randint(0, 10_000, (n,), generator=g, device="cuda", dtype=TORCH[dtype]), int(round(keep * 10_000))
    return torch.rand(n, generator=g, device="cuda", dtype=TORCH[dtype]), float(keep)


def _null_words(flags):
    """Flags as the reference's bit-packed null mask."""
    n = flags.numel()
    padded = torch.zeros((n + 63) // 64 * 64, dtype=torch.bool, device="cuda")
    padded[:n] = flags
    bits = torch.arange(8, dtype=torch.uint8, device="cuda")
    return (padded.view(-1, 8).to(torch.uint8) << bits).sum(1, dtype=torch.uint8).view(torch.int64)


def _columns(case, seed):
    """The case's columns and what they were made from."""
    g, n, kind = _gen(seed), case["rows"], case["kind"]
    if kind == "groupby":
        c = {"ranks": _ranks(g, n, case["groups"], case["skew"])}
        c["keys"] = _key_of(c["ranks"], case["keys"], case["spread"])
        c["vals"] = _values(g, n, case["vals"])
        if case["pred"]:
            c["filter"], c["below"] = _filter_column(g, n, case["pred"], case["keep"])
            c["filter"][_once(n, case["groups"])] = 0
    elif kind == "composite":
        side = case["side"]
        pair = _ranks(g, n, side * side, 0.0)
        c = {"k0": (pair // side).to(torch.int32), "k1": (pair % side).to(torch.int32), "vals": _values(g, n, "int64")}
    elif kind == "nulls":
        c = {"ranks": _ranks(g, n, case["groups"], 0.0), "vals": _values(g, n, case["vals"])}
        c["keys"] = _key_of(c["ranks"], "int32", True)
        c["key_null"] = torch.rand(n, generator=g, device="cuda") < 0.05
        c["val_null"] = torch.rand(n, generator=g, device="cuda") < 0.10
        c["key_null"][_once(n, case["groups"])] = False
        c["val_null"][_once(n, case["groups"])] = False
    elif kind == "compacted":
        c = {"ranks": _ranks(g, n, case["groups"], 0.0), "vals": _values(g, n, "int32")}
        c["keys"] = _key_of(c["ranks"], "int64", True)
        c["filter"], c["below"] = _filter_column(g, n, "int32", case["keep"])
        c["filter"][_once(n, case["groups"])] = 0
    elif kind == "order_by":
        c = {"amount": torch.round(_values(g, n, "float64") * 100) / 100,
             "region": torch.randint(0, case["regions"], (n,), generator=g, device="cuda", dtype=torch.int32)}
    else:  # scalar
        c = {"vals": _values(g, n, case["vals"])}
        c["filter"], c["below"] = _filter_column(g, n, "float32", case["keep"])
    return c


def _strings(case, seed):
    """A GPUString column: each row one of `groups` distinct strings of 8 to `longest` bytes, Zipf(1.1)."""
    g, d, longest = _gen(seed), case["groups"], case["longest"]
    ids = torch.arange(d, device="cuda")
    lens = 8 + (ids * 7919) % (longest - 7)
    text = torch.full((d, longest), ord("#"), dtype=torch.uint8, device="cuda")
    text[:, 0] = ord("c")
    for j in range(7):
        text[:, 1 + j] = (ord("0") + (ids // 10 ** (6 - j)) % 10).to(torch.uint8)
    pick = _ranks(g, case["rows"], d, 1.1)
    # Sums of values this wide do not tie, so ORDER BY SUM gives one order.
    vals = torch.randint(-(1 << 50), 1 << 50, (case["rows"],), generator=g, device="cuda")
    ends = torch.cumsum(lens[pick], 0)
    chars = torch.cat([text[p][torch.arange(longest, device="cuda") < lens[p][:, None]] for p in pick.split(1 << 22)])
    return {"pick": pick, "text": text, "lens": lens, "vals": vals, "chars": chars, "ends": ends}


def _batch_shapes(case):
    """Rows (least to most, even over their logarithm), groups and value type of every query."""
    q = case["queries"]
    out = []
    for i in range(q):
        rows = int(round(case["least"] * (case["most"] / case["least"]) ** (i / max(q - 1, 1))))
        groups = int(round(4 * min(16384.0, rows / 16) ** (((i * 7) % q) / max(q - 1, 1))))
        out.append((rows, groups, ("int64", "float32")[i % 2]))
    return out


def _aggs(case):
    return case["aggs"].split(",")


def prepare(case, seed):
    """Columns, and the table (or batch) that the program keeps between queries."""
    kind = case["kind"]
    if kind == "batch":
        g, queries = _gen(seed), []
        for rows, groups, vals in _batch_shapes(case):
            k = _ranks(g, rows, groups, 0.0).to(torch.int32)
            v = _values(g, rows, vals)
            queries.append(Query(k, v, ["sum", "max", "count"], max_groups=groups))
        tables, results = required_bytes(queries)
        b = GroupByBatch(len(queries), tables + (1 << 20), results + (1 << 20))
        b.set(queries)
        return {"case": case, "batch": b}
    if kind == "strings":
        c = _strings(case, seed)
        t = gb.StringGroupByTable(["sum", "count"], np.int64, case["groups"])
        return {"case": case, "keys": gb.GPUString(c["chars"], c["ends"]), "vals": c["vals"], "table": t}
    c = _columns(case, seed)
    s = {"case": case, **{k: v for k, v in c.items() if k not in ("ranks", "key_null", "val_null")}}
    if kind == "groupby":
        s["pred"] = gb.make_pred(c["filter"], F.less, c["below"], NUMPY[case["pred"]]) if case["pred"] else None
        s["bound"] = case["mod"] * 2 if case["mod"] else case["groups"]  # the remainder has the key's sign
        if not case["fresh"]:
            s["table"] = gb.GroupByTable(_aggs(case), NUMPY[case["keys"]], NUMPY[case["vals"]], s["bound"])
    elif kind == "composite":
        s["table"] = gb.GroupByTable(["sum", "count", "max"], np.int32, np.int64, case["side"] ** 2, n_key_cols=2)
    elif kind == "nulls":
        s["key_nulls"], s["val_nulls"] = _null_words(c["key_null"]), _null_words(c["val_null"])
        s["table"] = gb.GroupByTable(["min", "max", "avg", "count"], np.int32, NUMPY[case["vals"]], case["groups"])
    elif kind == "compacted":
        s["table"] = gb.GroupByTable(["sum", "count"], np.int64, np.int32, case["groups"])
    elif kind == "scalar":
        s["pred"] = gb.make_pred(c["filter"], F.less, c["below"], np.float32)
        s["acc"] = gb.ScalarAggregate(NUMPY[case["vals"]])
    return s


# ---------------------------------------------------------------------------------------------------------------
# One pass.
# ---------------------------------------------------------------------------------------------------------------
def _take(buf, perm):
    src = buf.torch() if isinstance(buf, gb.DeviceBuffer) else buf
    out = torch.empty_like(src)
    gb.GPUOrderBy.ReOrderByIdx(out, perm, src, src.numel())
    return out


def _ordered(table, aggs=None):
    """GetResults ORDER BY the keys: the key columns, then every aggregate."""
    keys, _, vals, n = table.results(aggs)
    cols = [k.torch() for k in keys]
    perm = gb.order_by(cols)
    return {"keys": [_take(k, perm) for k in cols], **{a: _take(v[0], perm) for a, v in vals.items()}}


def run(s):
    case = s["case"]
    return globals()["_run_" + case["kind"]](case, s)


def _run_groupby(case, s):
    if case["fresh"]:
        t = gb.GroupByTable(_aggs(case), NUMPY[case["keys"]], NUMPY[case["vals"]], s["bound"])
    else:
        t = s["table"]
        t.reset()
    if case["mod"]:
        gb.process_mod(t, s["keys"], case["mod"], s["vals"], s["pred"])
    else:
        t.process(s["keys"], s["vals"], pred=s["pred"])
    return _ordered(t)


def _run_composite(case, s):
    t = s["table"]
    t.reset()
    t.process([s["k0"], s["k1"]], s["vals"])
    return _ordered(t)


def _run_nulls(case, s):
    t = s["table"]
    t.reset()
    t.process(s["keys"], s["vals"], key_nulls=s["key_nulls"], value_nulls=s["val_nulls"])
    keys, knulls, vals, n = t.results()
    k, kn = keys[0].torch(), knulls[0].torch()
    perm = gb.order_by([k], nulls=[kn])  # the NULL group first
    words = torch.empty_like(kn)
    gb.GPUOrderBy.ReOrderNullValuesByIdx(words, perm, kn, n)
    return {"keys": _take(k, perm), "key_nulls": words, **{a: _take(v[0], perm) for a, v in vals.items()}}


def _run_compacted(case, s):
    n, t = case["rows"], s["table"]
    t.reset()
    mask = torch.empty(n, dtype=torch.int8, device="cuda")
    gb.GPUBinary.Binary(F.less, mask, s["filter"], np.int32(s["below"]), n)
    keys, m, _ = gb.GPUReconstruct.reconstructColKeep(s["keys"], mask, n)
    vals, _, _ = gb.GPUReconstruct.reconstructColKeep(s["vals"], mask, n)
    t.process(keys, vals, n=m)
    return _ordered(t)


def _run_strings(case, s):
    t = s["table"]
    t.reset()
    t.process(s["keys"], s["vals"])
    keys, _, vals, n = t.results()
    total = vals["sum"][0].torch()
    perm = gb.order_by([total], descending=[True])
    # The keys in that order, one row of `longest` bytes each, zero beyond their end.
    chars, ends = keys.allChars.torch(), keys.stringIndices.torch()
    lens = torch.diff(ends, prepend=ends.new_zeros(1))
    first, lens = _take(ends - lens, perm), _take(lens, perm)
    col = torch.arange(case["longest"], device="cuda")
    text = chars[(first[:, None] + col).clamp_(max=chars.numel() - 1)] * (col < lens[:, None])
    return {"keys": text, "lens": lens, "sum": _take(total, perm), "count": _take(vals["count"][0], perm)}


def _run_order_by(case, s):
    perm = gb.order_by([s["amount"], s["region"]], descending=[True, False])
    return {"rows": perm, "amount": _take(s["amount"], perm)}


def _run_scalar(case, s):
    s["acc"].reset()
    s["acc"].process(s["vals"], pred=s["pred"])
    return [s["acc"].result(a) for a in ("count", "sum", "avg", "min", "max")]


def _run_batch(case, s):
    b = s["batch"]
    b.run(graph=True)
    b.fetch()
    cols = {"keys": [], "count": [], "isum": [], "imax": [], "fsum": [], "fmax": []}
    for r in b.results_all():
        at = np.argsort(r["keys"][0])
        whole = r["sum"].dtype.kind == "i"
        cols["keys"].append(r["keys"][0][at])
        cols["count"].append(r["count"][at])
        cols["isum" if whole else "fsum"].append(r["sum"][at])
        cols["imax" if whole else "fmax"].append(r["max"][at])
    return {k: np.concatenate(v) for k, v in cols.items()}


# ---------------------------------------------------------------------------------------------------------------
# What a pass cannot do without: each input read once, each output written once.
# ---------------------------------------------------------------------------------------------------------------
def _agg_bytes(aggs, vals):
    return sum(8 if a == "count" else SIZE[vals] for a in aggs)


def work(case):
    n, kind = case.get("rows", 0), case["kind"]
    if kind == "groupby":
        read = SIZE[case["keys"]] + (SIZE[case["vals"]] if case["aggs"] != "count" else 0) + SIZE.get(case["pred"], 0)
        groups = min(n, case["mod"] or case["groups"])
        write = SIZE[case["keys"]] + _agg_bytes(_aggs(case), case["vals"])
        return {"bytes": n * read + groups * write, "flops": n}
    if kind == "composite":
        return {"bytes": n * 16 + min(n, case["side"] ** 2) * 32, "flops": n}
    if kind == "nulls":
        size = SIZE[case["vals"]]
        return {"bytes": n * (4 + size) + n // 4 + case["groups"] * (12 + 3 * size), "flops": n}
    if kind == "compacted":
        return {"bytes": n * 4 + int(n * case["keep"]) * 12 + case["groups"] * 20, "flops": n}
    if kind == "strings":
        mean = 8 + (case["longest"] - 8) / 2
        return {"bytes": int(n * (mean + 16) + case["groups"] * (case["longest"] + 24)), "flops": n}
    if kind == "order_by":
        return {"bytes": n * (12 + 4 + 8), "flops": n}
    if kind == "scalar":
        return {"bytes": n * (4 + SIZE[case["vals"]]), "flops": n}
    return {"bytes": sum(r * (4 + SIZE[v]) + g * (20 + SIZE[v]) for r, g, v in _batch_shapes(case)), "flops": 0}


def tolerance(case):
    """Whole numbers, MIN and MAX are the same; float sums and averages are correct to the rounding of their type (a
    32-bit result is a 64-bit sum rounded once: half a unit in the last place, 6e-8, seen from either side).  Without
    NULLs a sum of doubles may be held in 64-bit fixed point that keeps 24 bits of the smallest addend."""
    kind, vals = case["kind"], case.get("vals")
    if kind in ("composite", "compacted", "strings", "order_by") or vals in ("int32", "int64"):
        return "exact"
    if vals == "float64":
        return {"rel": 1e-12, "max": 1e-10} if kind == "groupby" else {"rel": 1e-13, "max": 1e-12}
    return {"rel": 1.5e-7, "max": 5e-7}


# ---------------------------------------------------------------------------------------------------------------
# The exact result in 64 bits, by group number.
# ---------------------------------------------------------------------------------------------------------------
def _by_group(ids, vals, groups, aggs):
    """Aggregates of `vals` per group number in [0, groups): 64-bit sums, and the C++ rules of the narrow types."""
    whole = not vals.is_floating_point()
    count = torch.bincount(ids, minlength=groups)
    out = {"n": count}
    if "count" in aggs:
        out["count"] = count
    if "sum" in aggs or "avg" in aggs:
        total = torch.zeros(groups, dtype=torch.int64 if whole else torch.float64, device="cuda")
        for i, v in zip(ids.split(1 << 26), vals.split(1 << 26)):
            total.index_add_(0, i, v.to(total.dtype))
        if whole:
            total = total.to(vals.dtype).to(torch.int64)  # an integer SUM wraps in the value type
        out["sum"] = total
        if "avg" in aggs:
            safe = count.clamp(min=1)
            out["avg"] = torch.div(total, safe, rounding_mode="trunc") if whole else total / safe
    for a, how in (("min", "amin"), ("max", "amax")):
        if a in aggs:
            out[a] = torch.zeros(groups, dtype=vals.dtype, device="cuda").scatter_reduce_(
                0, ids, vals, how, include_self=False)
    return out


def _sorted_rows(keys, cols, present):
    """The rows of the groups that are present, ordered by `keys`."""
    rows = present.nonzero().view(-1)
    rows = rows[torch.argsort(keys[rows])]
    return keys[rows], {a: c[rows] for a, c in cols.items()}


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return None  # the batch's own single queries are the other cases' shapes
    if kind == "strings":
        c = _strings(case, seed)
        r = _by_group(c["pick"], c["vals"], case["groups"], ["sum", "count"])
        rows = (r["n"] > 0).nonzero().view(-1)
        rows = rows[torch.argsort(r["sum"][rows], descending=True)]
        col = torch.arange(case["longest"], device="cuda")
        return {"keys": c["text"][rows] * (col < c["lens"][rows][:, None]), "lens": c["lens"][rows],
                "sum": r["sum"][rows], "count": r["count"][rows]}
    c = _columns(case, seed)
    if kind == "order_by":
        perm = torch.sort(c["region"], stable=True).indices
        perm = perm[torch.sort(c["amount"][perm], descending=True, stable=True).indices]
        return {"rows": perm.to(torch.int32), "amount": c["amount"][perm]}
    keep = c["filter"] < torch.tensor(c["below"], dtype=c["filter"].dtype) if "filter" in c else None
    if kind == "scalar":
        v = c["vals"][keep]
        if not v.is_floating_point():
            total = int(v.to(torch.int64).sum())
            total = (total + (1 << 31)) % (1 << 32) - (1 << 31) if v.dtype == torch.int32 else total
            return [v.numel(), total, int(total / v.numel()) if abs(total) < 1 << 50 else None, int(v.min()), int(v.max())]
        total = float(v.double().sum())
        return [v.numel(), total, total / v.numel(), float(v.min()), float(v.max())]
    if kind == "composite":
        side = case["side"]
        ids = c["k0"].to(torch.int64) * side + c["k1"]
        r = _by_group(ids, c["vals"], side * side, ["sum", "count", "max"])
        ids, cols = _sorted_rows(torch.arange(side * side, device="cuda"), r, r["n"] > 0)
        return {"keys": [ids // side, ids % side], **{a: cols[a] for a in ("sum", "count", "max")}}
    ids, vals = c["ranks"], c["vals"]
    if kind == "nulls":
        groups = case["groups"]
        ids = torch.where(c["key_null"], groups, ids)  # the NULL keys are one group, first in the order
        live = ~c["val_null"]
        seen = torch.bincount(ids, minlength=groups + 1) > 0
        r = _by_group(ids[live], vals[live], groups + 1, ["min", "max", "avg", "count"])
        keys = _key_of(torch.arange(groups + 1, device="cuda"), "int32", True).to(torch.int64)
        keys[groups] = -(1 << 40)
        keys, cols = _sorted_rows(keys, r, seen)
        return {"keys": torch.where(keys == -(1 << 40), 0, keys), "key_nulls": _null_words(keys == -(1 << 40)),
                **{a: cols[a] for a in ("min", "max", "avg", "count")}}
    if keep is not None:
        ids, vals = ids[keep], vals[keep]
    aggs, groups = (_aggs(case), case["groups"]) if kind == "groupby" else (["sum", "count"], case["groups"])
    if case.get("mod"):
        m = case["mod"]
        ids = torch.fmod(_key_of(ids, "int64", case["spread"]), m) + m  # C++ remainder: -m < r < m
        groups, keys = 2 * m, torch.arange(2 * m, device="cuda") - m
    else:
        keys = _key_of(torch.arange(groups, device="cuda"), case.get("keys", "int64"), case.get("spread", True))
    r = _by_group(ids, vals, groups, aggs)
    keys, cols = _sorted_rows(keys, r, r["n"] > 0)
    return {"keys": [keys], **{a: cols[a] for a in aggs}}
