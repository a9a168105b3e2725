"""The fast aggregation pass over NULL masks and row masks (single keys), against the oracle: every key and value type
at the edges of its 2048-row tile, tables that hold every group and tables that spill, keys that share the NULL key's
or the empty slot's word, groups without a non-NULL value, and the accuracy of SUM and AVG of doubles."""
import subprocess
import sys

import numpy as np
import pytest
import torch

from conftest import ROOT
from gpu_compare import FLOAT_RTOL
from qikkdb_b200.groupby import FilterConditions, GroupByTable, device_nullmask
from test_gpu_parity import ALL, _dev, run_both

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _fast_pass(monkeypatch):
    """The fast pass takes every masked call that it can, also those that the general one is picked for."""
    monkeypatch.setenv("QDB_AGG_FAST", "2")


def _keys(rng, n, groups, dt):
    k = rng.integers(0, groups, n)
    if dt in (np.float32, np.float64):
        k = k.astype(dt) * dt(0.25)
        k[rng.random(n) < 0.02] = dt(-0.0)
        return k
    k = (k * (0x9E3779B1 if dt == np.int32 else 0x1234567)).astype(dt)
    lowest = np.iinfo(dt).min
    for x in (lowest, lowest + 1):  # int64: the empty slot's word and the NULL key's
        k[rng.random(n) < 0.01] = x
    return k


def _vals(rng, n, dt):
    if dt in (np.float32, np.float64):
        v = np.exp(rng.standard_normal(n) + 2).astype(dt)
        v[rng.random(n) < 0.01] *= dt(1e12)  # outside the fixed-point window
        return v
    return rng.integers(-(1 << 30), 1 << 30, n).astype(dt)


@pytest.mark.parametrize("n", [2047, 2048, 2049, 6145, 303_103, 1_500_001])
@pytest.mark.parametrize("kdt", [np.int32, np.int64, np.float32, np.float64])
@pytest.mark.parametrize("vdt", [np.int32, np.int64, np.float32, np.float64])
@pytest.mark.parametrize("groups", [37, 60_000])
def test_masked_groupby(cuda, n, kdt, vdt, groups):
    if n > 303_103 and (kdt, vdt) not in ((np.int64, np.float64), (np.int32, np.int64)):
        pytest.skip("the largest size for two type pairs")
    rng = np.random.default_rng([n, groups, np.dtype(kdt).num, np.dtype(vdt).num])
    k, v = _keys(rng, n, groups, kdt), _vals(rng, n, vdt)
    kn, vn = rng.random(n) < 0.1, (rng.random(n) < 0.3) | (k == k[0])  # the group of k[0] has no value
    vf, kf = vdt in (np.float32, np.float64), kdt in (np.float32, np.float64)
    v = v.copy()
    if vf:
        v[vn] = np.nan  # what a NULL row holds must not matter
    pt = (np.int32, np.int64, np.float32, np.float64)[n % 4]
    pcol = rng.integers(0, 100, n).astype(pt)
    pred = (pcol, FilterConditions.less, 60, np.int32, rng.random(n) < 0.05)
    mask = (rng.random(n) < 0.8).astype(np.int8)
    cap = groups + 3
    kw = dict(val_is_float=vf, key_is_float=kf)
    run_both(k, v, ALL, cap, key_nulls=[kn], val_nulls=vn, pred=pred, mask=mask, **kw)
    run_both(k, v, ["sum"], cap, key_nulls=[kn], val_nulls=vn, **kw)
    run_both(k, v, ["min", "max"], cap, val_nulls=vn, blocks=3 if n > 10_000 else 1, **kw)
    run_both(k, v, ["count"], cap, val_nulls=vn, pred=pred, **kw)
    run_both(k, np.where(vn, v.dtype.type(1), v), ["sum", "max"], cap, key_nulls=[kn], mask=mask, **kw)


def test_masked_all_rows_null_or_filtered(cuda):
    n = 10_000
    k = np.arange(n, dtype=np.int64)
    v = np.ones(n)
    run_both(k, v, ALL, n + 1, key_nulls=[np.ones(n, bool)], val_is_float=True)
    run_both(k, v, ALL, n + 1, val_nulls=np.ones(n, bool), val_is_float=True)
    run_both(k, v, ALL, n + 1, mask=np.zeros(n, np.int8), val_is_float=True)


@pytest.mark.parametrize("groups", [50, 40_000])
def test_masked_double_sums(cuda, groups):
    """Doubles under NULL masks are summed in 96-bit fixed point: within 2^-62 of the first tile's largest value per
    addend, or 2^-49 of it for the few above 2^2 times that.  Partial sums meet in FP64 atomics (at most 148 CTAs' per
    group), so the relative error of a sum of positive values of like size stays below 148 x 2^-53 + 2^-49."""
    n = 2_000_003
    rng = np.random.default_rng(groups)
    k = rng.integers(0, groups, n)
    v = np.exp(rng.standard_normal(n) + 2)
    vn = rng.random(n) < 0.2
    rel, _, _ = run_both(k, v, ["sum", "avg"], groups, val_nulls=vn, val_is_float=True)
    assert rel <= 1e-12 < FLOAT_RTOL


@pytest.mark.parametrize("groups", [10, 400, 20_000])
@pytest.mark.parametrize("stride", [1, 0x9E3779B97F4A7C15 - (1 << 64), 86_400_000_000])
def test_evenly_spaced_keys(cuda, groups, stride):
    """Keys in arithmetic progression, one stride of which crowds the table's home buckets (the multiplicative hash is
    linear), in tables that hold every group and in spilled partitions; few groups hold copies of every state."""
    n = 600_011
    rng = np.random.default_rng(groups)
    with np.errstate(over="ignore"):
        k = rng.integers(0, groups, n).astype(np.int64) * np.int64(stride)
    run_both(k, rng.integers(-1000, 1000, n).astype(np.int32), ALL, groups)
    run_both(k, np.exp(rng.standard_normal(n)).astype(np.float32), ["sum", "max"], groups, val_is_float=True)


def _growing(n, groups, dt, rng):
    """A column whose first tiles hold values of about 1 and whose later rows, two by two in one group, hold v and its
    negative, v up to 2^14, beside values of about 2^-22: every group's sum is a sum of the small ones alone.  All
    values are multiples of 2^-46 and exact in either type."""
    k = np.repeat(rng.integers(0, groups, (n + 3) // 4), 4)[:n].astype(np.int32)
    v = np.empty(n, dtype=np.float64)
    first = 148 * 2048
    quad = np.arange(n) % 4
    size = np.exp2(rng.integers(2, 14, (n + 3) // 4).astype(np.float64)).repeat(4)[:n]
    size *= (1 + rng.integers(0, 1 << 23, (n + 3) // 4) / (1 << 23)).repeat(4)[:n]
    small = (1 + rng.integers(0, 1 << 23, n) / (1 << 23)) * 2.0 ** -23
    v = np.where(quad == 0, size, np.where(quad == 1, -size, small))
    head = (1 + rng.integers(0, 1 << 20, (n + 3) // 4) / (1 << 20)).repeat(4)[:n]
    head = np.where(quad % 2 == 0, head, -head)
    v[:first] = head[:first]
    return k, v.astype(dt)


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("groups", [10, 2000])
def test_masked_sums_of_growing_columns(cuda, groups, dt):
    """Values far above and below those of a CTA's first tile (2^15 times up, 2^-23 down) stay in the 96-bit sums, which
    are exact here, whatever the order: a row added in FP64 instead would leave its rounding at 2^14's last place."""
    n = 1_600_000
    rng = np.random.default_rng(groups)
    k, v = _growing(n, groups, dt, rng)
    vn = np.zeros(n, bool)
    vn[rng.integers(148 * 2048 // 4, n // 4, n // 50) * 4 + 2] = True  # small ones: sums stay below 2^53 units of 2^-46
    t = GroupByTable(["sum"], np.int32, dt, groups)
    t.process([_dev(k)], _dev(v), n, None, device_nullmask(vn))
    r = t.results_numpy()
    ints = np.where(vn, 0, np.round(v.astype(np.float64) * 2.0 ** 46)).astype(np.int64)  # exact: below 2^61
    exp = np.zeros(groups, dtype=np.int64)
    np.add.at(exp, k, ints)
    order = np.argsort(r["keys"][0])
    keys = r["keys"][0][order]
    assert len(keys) == len(np.unique(k))
    assert (r["sum"][order] == (exp[keys].astype(np.float64) * 2.0 ** -46).astype(dt)).all()


@pytest.mark.parametrize("dt", [np.float32, np.float64])
def test_masked_growing_column_stays_on_chip(cuda, monkeypatch, dt):
    """A column that grows 2^12-fold along its rows, 10 groups: no slower than the general pass (rows that leave the
    fixed-point window would be added to ten words of the global table)."""
    n = 1 << 23
    g = torch.Generator(device="cuda").manual_seed(1)
    k = torch.randint(0, 10, (n,), generator=g, device="cuda", dtype=torch.int32)
    tt = torch.float32 if dt == np.float32 else torch.float64
    v = torch.rand(n, generator=g, device="cuda", dtype=tt) + torch.arange(n, device="cuda", dtype=tt) * (4096.0 / n)
    null = torch.zeros(n // 64, dtype=torch.int64, device="cuda")
    null[::3] = 5
    t = GroupByTable(["sum"], np.int32, dt, 10)
    us = {}
    for fast in ("1", "0"):
        monkeypatch.setenv("QDB_AGG_FAST", fast)
        best = float("inf")
        for _ in range(4):
            t.reset()
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            t.process([k], v, n, None, null, sync=False)
            e[1].record()
            torch.cuda.synchronize()
            best = min(best, e[0].elapsed_time(e[1]) * 1e3)
        us[fast] = best
    assert us["1"] <= 1.25 * us["0"], us  # a quarter for the measurement; 67 times as long when rows leave the window


@pytest.mark.parametrize("n,groups,dt,aggs,what", [
    (100_000, 3000, torch.int32, ["sum", "count"], "values"), (2_000_000, 3000, torch.float64, ["sum"], "values"),
    (4_000_000, 2_000_000, torch.float64, ["min", "max", "sum", "count"], "rows"),
    (16_000_000, 4, torch.int32, ["sum"], "rows"), (1_000_000, 30_000, torch.int64, ["sum"], "values"),
    (16_000_000, 100_000, torch.float64, ["max", "avg"], "keys")])
def test_masked_calls_take_the_faster_pass(cuda, monkeypatch, n, groups, dt, aggs, what):
    """Which pass takes a masked call: not slower than either of them (a fifth for the measurement)."""
    g = torch.Generator(device="cuda").manual_seed(1)
    k = torch.randint(0, groups, (n,), generator=g, device="cuda", dtype=torch.int32)
    v = (torch.rand(n, generator=g, device="cuda") * 1000).to(dt)
    nulls = torch.randint(-(1 << 63), (1 << 63) - 1, ((n + 63) // 64,), generator=g, device="cuda")
    kw = {"values": dict(value_nulls=nulls), "keys": dict(key_nulls=[nulls]),
          "rows": dict(mask=(torch.rand(n, generator=g, device="cuda") < 0.5).to(torch.int8))}[what]
    t = GroupByTable(aggs, np.int32, {torch.int32: np.int32, torch.int64: np.int64, torch.float64: np.float64}[dt], groups)
    us = {}
    for fast in ("1", "0", "2"):
        monkeypatch.setenv("QDB_AGG_FAST", fast)
        us[fast] = float("inf")
        for _ in range(6):
            t.reset()
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            t.process([k], v, n, sync=False, **kw)
            e[1].record()
            torch.cuda.synchronize()
            us[fast] = min(us[fast], e[0].elapsed_time(e[1]) * 1e3)
    assert us["1"] <= 1.2 * min(us.values()) + 3, us


_TIGHT = """
import numpy as np, os, torch
from qikkdb_b200.groupby import GroupByTable
n, groups = 1 << 26, 100_000
g = torch.Generator(device="cuda").manual_seed(1)
k = torch.randint(0, groups, (n,), generator=g, device="cuda", dtype=torch.int32)
v = torch.randint(-1000, 1000, (n,), generator=g, device="cuda")
mask = (torch.rand(n, generator=g, device="cuda") < 0.5).to(torch.int8)
t = GroupByTable(["sum", "count"], np.int32, np.int64, groups)
exp = torch.zeros(groups, dtype=torch.int64, device="cuda").index_add_(0, k.long(), v * mask)
torch.cuda.synchronize()
torch.cuda.empty_cache()
free, _ = torch.cuda.mem_get_info()
hog = torch.empty(free - (1 << 30), dtype=torch.uint8, device="cuda")  # leaves 1 GiB
t.process([k], v, n, mask=mask)
del hog
torch.cuda.empty_cache()
r = t.results_numpy()
o = np.argsort(r["keys"][0])
assert (r["sum"][o] == exp.cpu().numpy()).all()
print("tight ok")
"""


def test_masked_call_with_little_memory(cuda):
    """A masked call of 2^26 rows that spills, with 1 GiB of memory left: the fast pass's spill area takes 1.3 GB, the general
    pass's 0.7, and the call is served as before."""
    res = subprocess.run([sys.executable, "-c", _TIGHT], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert res.returncode == 0 and "tight ok" in res.stdout, res.stdout + res.stderr
