"""The fast aggregation pass over NULL masks and row masks (single keys), against the oracle: every key and value type
at the edges of its 2048-row tile, tables that hold every group and tables that spill, keys that share the NULL key's
or the empty slot's word, groups without a non-NULL value, and the accuracy of SUM and AVG of doubles."""
import numpy as np
import pytest

from gpu_compare import FLOAT_RTOL
from qikkdb_b200.groupby import FilterConditions
from test_gpu_parity import ALL, run_both

pytestmark = pytest.mark.gpu


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
    """Doubles under NULL masks are summed in 96-bit fixed point: 2^-62 of the largest value per addend.  Partial sums
    meet in FP64 atomics (at most 148 CTAs' per group), so the relative error of a sum of positive values of like size
    stays below 148 x 2^-53 + the window's 2^-40 for the smallest values it keeps."""
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
