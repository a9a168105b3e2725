"""ORDER BY of GROUP BY results on the GPU (qdb_order_by_column / qdb_order_by / qdb_reorder, the replacement of
GPUOrderBy, qikkDB/QueryEngine/GPUCore/GPUOrderBy.cuh:88-195) against the oracle: the reference's GROUP BY +
ORDER BY known answers, then random multi-column orders with NULLs, ties, descending columns, IEEE edge values and
row counts around a tile, OFFSET / LIMIT through the gather, and an ORDER BY of the 16.8M-group result
of the composite-key GROUP BY.  Permutations must equal the oracle's exactly (the sort is stable)."""
import json
import os

import numpy as np
import pytest
import torch

import oracle
from qikkdb_b200 import datagen as dg
from qikkdb_b200.groupby import GPUOrderBy, GroupByTable, order_by, pack_nullmask, unpack_nullmask

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def test_group_by_order_by_reference_kats(cuda):
    """DispatcherGroupByTests.cpp:1551-1588 through the operator mirror: GROUP BY on the GPU, then GPUOrderBy
    OrderByColumn + ReOrderByIdx over the result columns, as the dispatcher runs them."""
    with open(os.path.join(HERE, "golden", "reference_kats.json")) as f:
        cases = json.load(f)["order_by_cases"]
    for c in cases:
        k = np.asarray(c["keys"], dtype=np.int32)
        v = np.asarray(c["values"], dtype=np.int32)
        t = GroupByTable(["sum"], np.int32, np.int32, 1024)
        t.process([_dev(k)], _dev(v), len(k))
        keys, _, vals, n = t.results(["sum"])
        kd, sd = keys[0].torch(), vals["sum"][0].torch()
        ob = GPUOrderBy(n)
        idx = torch.empty(n, dtype=torch.int32, device="cuda")
        ob.OrderByColumn(idx, kd if c["order_by"] == "key" else sd, None, n,
                         GPUOrderBy.DESC if c["descending"] else GPUOrderBy.ASC)
        ok, os_ = torch.empty_like(kd), torch.empty_like(sd)
        GPUOrderBy.ReOrderByIdx(ok, idx, kd, n)
        GPUOrderBy.ReOrderByIdx(os_, idx, sd, n)
        got = [[int(a), int(b)] for a, b in zip(ok.cpu().numpy(), os_.cpu().numpy())]
        assert got == c["expected"], (c["name"], got)


def _random_cols(rng, n, spec):
    cols, nulls = [], []
    for dt, card, null_frac in spec:
        if dt in (np.float32, np.float64):
            x = rng.integers(-card, card, n).astype(dt) * dt(0.5)
            edge = np.array([0.0, -0.0, np.inf, -np.inf, np.finfo(dt).max, -np.finfo(dt).max], dtype=dt)
            pick = rng.random(n) < 0.05
            x[pick] = edge[rng.integers(0, len(edge), int(pick.sum()))]
        else:
            x = rng.integers(-card, card, n).astype(dt)
            pick = rng.random(n) < 0.01
            x[pick] = np.iinfo(dt).min
        cols.append(x)
        nulls.append(pack_nullmask(rng.random(n) < null_frac) if null_frac > 0 else None)
    return cols, nulls


@pytest.mark.parametrize("n", [0, 1, 2047, 2048, 2049, 100_003])
def test_order_by_random_against_oracle(cuda, n):
    rng = np.random.default_rng(n + 7)
    spec = [(np.int32, 50, 0.05), (np.float64, 1000, 0.0), (np.int64, 1 << 40, 0.1), (np.float32, 30, 0.02)]
    cols, nulls = _random_cols(rng, n, spec)
    desc = [False, True, False, True]
    exp = oracle.order_by(cols, desc, nulls)
    got = order_by([_dev(c) for c in cols], desc,
                   [None if x is None else _dev(x.view(np.int64)) for x in nulls]).cpu().numpy()
    assert (got == exp).all()


def test_order_by_offset_limit_and_nulls(cuda):
    rng = np.random.default_rng(11)
    n = 50_000
    v = rng.integers(-1000, 1000, n).astype(np.int32)
    nflags = rng.random(n) < 0.1
    nw = pack_nullmask(nflags)
    exp = oracle.order_by([v], [True], [nw])
    idx = order_by([_dev(v)], [True], [_dev(nw.view(np.int64))])
    offset, limit = 123, 4567
    out = torch.empty(limit, dtype=torch.int32, device="cuda")
    GPUOrderBy.ReOrderByIdx(out, idx, _dev(v), limit, offset=offset)
    assert (out.cpu().numpy() == v[exp[offset:offset + limit]]).all()
    onull = torch.zeros((limit + 63) // 64, dtype=torch.int64, device="cuda")
    GPUOrderBy.ReOrderNullValuesByIdx(onull, idx, _dev(nw.view(np.int64)), limit, offset=offset)
    assert (unpack_nullmask(onull.cpu().numpy(), limit) == nflags[exp[offset:offset + limit]]).all()


def test_order_by_composite_groupby_results(cuda):
    """ORDER BY SUM DESC, key0, key1 over the 16.8M groups of a 2^26-row composite-key GROUP BY."""
    n = 1 << 26
    a = dg.uniform_i32(43, 0, n, 0, 4095)
    b = dg.uniform_i32(43, 1, n, 0, 4095)
    v = dg.uniform_i64(43, 2, n, 0, (1 << 31) - 1)
    t = GroupByTable(["sum"], np.int32, np.int64, 1 << 24, n_key_cols=2)
    t.process([_dev(a), _dev(b)], _dev(v), n)
    keys, _, vals, g = t.results(["sum"])
    k0, k1, s = keys[0].torch(), keys[1].torch(), vals["sum"][0].torch()
    idx = order_by([s, k0, k1], [True, False, False]).cpu().numpy()
    exp = oracle.order_by([s.cpu().numpy(), k0.cpu().numpy(), k1.cpu().numpy()], [True, False, False])
    assert g > 10_000_000 and (idx == exp).all()


@pytest.mark.parametrize("n", [1, 31, 255, 257, 4095, 4096, 4097, 6144, 8191, 8192, 8193, 12_289, 300_007])
@pytest.mark.parametrize("shape", ["constant", "one_digit", "wide", "columns"])
def test_order_by_forms_and_skipped_digits(cuda, n, shape):
    """Both forms of the sort (one block up to 8192 rows, tiles of 4096 64-bit or 6144 32-bit keys above) at the edges
    of their tiles, with digits that are the same in every row (passes that do not run, in any place of the order,
    or all of them) and more columns than one launch of the one-block form takes."""
    rng = np.random.default_rng(n)
    nulls = None
    if shape == "constant":
        cols = [np.full(n, 7, np.int64), np.full(n, -3, np.int32)]
    elif shape == "one_digit":
        cols = [(rng.integers(0, 256, n).astype(np.int64) << 40) + 5, (rng.integers(0, 3, n) << 8).astype(np.int32)]
    elif shape == "wide":
        cols = [rng.integers(-(1 << 62), 1 << 62, n), rng.standard_normal(n).astype(np.float32)]
        nulls = [pack_nullmask(rng.random(n) < 0.3), None]
    else:
        cols = [rng.integers(0, 2, n).astype(np.int32 if i % 2 else np.float64) for i in range(11)]
    desc = [bool(i % 2) for i in range(len(cols))]
    exp = oracle.order_by(cols, desc, nulls if nulls else [None] * len(cols))
    got = order_by([_dev(c) for c in cols], desc,
                   [None if x is None else _dev(x.view(np.int64)) for x in nulls] if nulls else None).cpu().numpy()
    assert (got == exp).all()
    # the same, column by column (the permutation is read back in)
    ob = GPUOrderBy(n)
    for i in reversed(range(len(cols))):
        ob.OrderByColumn(None, _dev(cols[i]), None if not nulls or nulls[i] is None else _dev(nulls[i].view(np.int64)),
                         n, int(desc[i]))
    assert (ob.indices[:n].cpu().numpy() == exp).all()


@pytest.mark.parametrize("n", [200, 9000])
def test_order_by_column_of_chosen_rows(cuda, n):
    """OrderByColumn over row numbers of a longer column (first == 0): both forms keep them whole."""
    from qikkdb_b200 import _capi as capi
    rng = np.random.default_rng(n)
    col = rng.integers(-50, 50, 300_000).astype(np.int32)
    rows = rng.permutation(len(col))[:n].astype(np.int32)
    idx, dc = _dev(rows), _dev(col)
    capi.check(capi.lib().qdb_order_by_column(capi.QDB_INT32, dc.data_ptr(), None, 0, n, 0, idx.data_ptr(),
                                              torch.cuda.current_stream().cuda_stream))
    assert (idx.cpu().numpy() == rows[np.argsort(col[rows], kind="stable")]).all()


@pytest.mark.parametrize("polls", [0, 3])
@pytest.mark.parametrize("dt", [np.int32, np.int64, np.float64])
def test_order_by_tiles_that_stop_waiting(cuda, monkeypatch, polls, dt):
    """A tile that has looked for its predecessors' counts in vain `polls` times counts their rows itself: with a limit of
    0 most tiles do, and the tiles behind them use what those publish."""
    monkeypatch.setenv("QDB_OB_POLLS", str(polls))
    n = 300_007
    rng = np.random.default_rng(polls)
    cols = [rng.integers(-1000, 1000, n).astype(np.int32), (rng.standard_normal(n) * 1e6).astype(dt)]
    exp = oracle.order_by(cols, [True, False], [None, None])
    dev = [_dev(c) for c in cols]
    for _ in range(5):
        assert (order_by(dev, [True, False], [None, None]).cpu().numpy() == exp).all()


@pytest.mark.parametrize("dt,most", [(np.int32, 13), (np.int64, 21)])
def test_order_by_scratch(cuda, dt, most):
    """Scratch of the tiled form: two key buffers, one of row numbers and half a byte of tile states a row."""
    from cuda.bindings import runtime as rt
    n = 3_000_000
    col = torch.from_numpy(np.random.default_rng(1).integers(-1 << 30, 1 << 30, n).astype(dt)).cuda()
    order_by([col], [False], [None])
    torch.cuda.synchronize()
    err, pool = rt.cudaDeviceGetDefaultMemPool(0)
    assert err == rt.cudaError_t.cudaSuccess
    attr = rt.cudaMemPoolAttr
    err, used = rt.cudaMemPoolGetAttribute(pool, attr.cudaMemPoolAttrUsedMemCurrent)
    assert err == rt.cudaError_t.cudaSuccess
    (err,) = rt.cudaMemPoolSetAttribute(pool, attr.cudaMemPoolAttrUsedMemHigh, type(used)(0))
    assert err == rt.cudaError_t.cudaSuccess
    idx = order_by([col], [False], [None])
    torch.cuda.synchronize()
    err, high = rt.cudaMemPoolGetAttribute(pool, attr.cudaMemPoolAttrUsedMemHigh)
    assert (torch.diff(col[idx.long()]) >= 0).all()
    assert 0 < int(high) - int(used) <= most * n
