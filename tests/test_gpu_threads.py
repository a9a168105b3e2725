"""Operators called from two host threads, each on a stream of its own (ctypes drops the interpreter's lock around a
call): a kernel's launch settings belong to the process, so no call may set them to what only its own sizes need."""
import threading

import numpy as np
import pytest
import torch

import oracle
from qikkdb_b200 import _capi as capi
from qikkdb_b200.groupby import GroupByTable, device_nullmask

pytestmark = pytest.mark.gpu


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _together(*jobs):
    """Runs the jobs in threads that start together, each in a stream of its own; re-raises the first error."""
    gate, errors = threading.Barrier(len(jobs)), []

    def body(job):
        try:
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                gate.wait()
                job()
                stream.synchronize()
        except BaseException as e:  # noqa: BLE001 - handed to the main thread
            errors.append(e)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=body, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if errors:
        raise errors[0]


def test_order_by_sizes_in_two_threads(cuda):
    """The one-block form of ORDER BY at two sizes, whose shared memory differs by a factor of two."""
    def job(n):
        col = np.random.default_rng(n).integers(-500, 500, n).astype(np.int32)
        dc, idx, lib = _dev(col), torch.empty(n, dtype=torch.int32, device="cuda"), capi.lib()

        def run():
            s = torch.cuda.current_stream().cuda_stream
            for _ in range(3000):
                capi.check(lib.qdb_order_by_column(capi.QDB_INT32, dc.data_ptr(), None, 0, n, 1, idx.data_ptr(), s))
        return run, idx, oracle.order_by([col], [False], [None])

    jobs = [job(8192), job(3000)]
    _together(*(j[0] for j in jobs))
    for _, idx, exp in jobs:
        assert (idx.cpu().numpy() == exp).all()


@pytest.mark.parametrize("kind,groups", [("few", (10, 5000)), ("masked", (50, 4000)), ("spilled", (60_000, 900_000)),
                                         ("general", (10, 4000))])
def test_group_by_tables_in_two_threads(cuda, kind, groups):
    """Every aggregation pass (without a ring, staged with NULL masks, spilling, and the general one that unaligned
    columns take) over tables of two sizes."""
    n = 20_001

    def job(g):
        rng = np.random.default_rng(g)
        k = rng.integers(0, min(g, n), n + 1).astype(np.int32)
        v = rng.integers(-1000, 1000, n + 1).astype(np.int32)
        off = 1 if kind == "general" else 0
        vn = rng.random(n) < 0.1 if kind == "masked" else None
        dk, dv, dn = _dev(k)[off:off + n], _dev(v)[off:off + n], device_nullmask(vn) if vn is not None else None
        t = GroupByTable(["sum", "max"], np.int32, np.int32, g)

        def run():
            for _ in range(500):
                t.reset()
                t.process([dk], dv, n, None, dn, sync=False)
        exp = {}
        for i in range(n):
            if vn is None or not vn[i]:
                x, y = int(k[off + i]), int(v[off + i])
                s, m = exp.get(x, (0, -1 << 40))
                exp[x] = (s + y, max(m, y))
        return run, t, exp

    jobs = [job(g) for g in groups]
    _together(*(j[0] for j in jobs))
    for _, t, exp in jobs:
        r = t.results_numpy()
        got = {int(k): (int(s), int(m)) for k, s, m, null in zip(r["keys"][0], r["sum"], r["max"], r["sum_null"])
               if not null}
        assert got == exp
