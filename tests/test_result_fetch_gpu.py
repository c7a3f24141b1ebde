"""Fetching result columns of few pages, which are in host memory already, and
of more: into pageable and page-locked buffers and page by page,
after later executions, with more results alive than the pool has buffers, with
more columns than a buffer holds, and from several threads."""
from __future__ import annotations

import ctypes as C
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def plan_of(hj, n, cols=3, seed=0, strings=True):
    r = np.random.default_rng(seed)
    cs = [hj.Column.int32(r.integers(-2**31, 2**31, n).astype(np.int32),
                          (r.random(n) < 0.9).astype(np.uint8) if k % 2 else None) for k in range(cols)]
    types = [hj.INT32] * cols
    if strings:
        lens = r.integers(0, 30, n)
        offs = np.zeros(n + 1, np.uint64)
        np.cumsum(lens, out=offs[1:])
        cs.append(hj.Column.varchar(r.integers(33, 127, max(1, int(offs[-1]))).astype(np.uint8), offs))
        types.append(hj.VARCHAR)
    p = hj.Plan()
    p.new_input(hj.Table(n, cs))
    p.root = p.new_scan_node(0, list(enumerate(types)))
    return p


def pages_of(hj, engine, r, col, how):
    import torch
    L, n = hj.lib(), C.c_uint64()
    assert L.hj_result_column(r, col, None, C.byref(n)) == 0
    n = int(n.value)
    if how == "pages":
        buf = np.zeros((n, hj.PAGE_SIZE), np.uint8)
        order = np.arange(n)[::-1]  # page i anywhere
        ptrs = (C.c_void_p * max(1, n))(*[buf[order[i]].ctypes.data for i in range(n)])
        assert L.hj_result_copy_pages(engine.handle, r, col, ptrs) == 0
        return buf[order]
    if how == "pageable":
        buf = np.zeros((n, hj.PAGE_SIZE), np.uint8)
        assert L.hj_result_copy_contiguous(engine.handle, r, col, buf.ctypes.data) == 0
        return buf
    t = torch.zeros((n, hj.PAGE_SIZE), dtype=torch.uint8)
    t = t.pin_memory() if how == "pinned" else t
    if n:
        assert L.hj_result_copy_contiguous(engine.handle, r, col, t.data_ptr()) == 0
    return t.numpy()


def check(hj, orc, engine, r, want, ncols, hows=("pages", "pageable", "pinned")):
    for how in hows:
        out = orc.Output(0, "", want.num_rows, [(want.columns[k][0], pages_of(hj, engine, r, k, how))
                                                for k in range(ncols)])
        a, b = orc.summary(out), orc.summary(want)
        assert a[:3] == b[:3] and np.array_equal(a[3], b[3]), how


@pytest.mark.parametrize("n", [0, 1, 1984, 8 * 1984, 8 * 1984 + 1, 60_000])
def test_sizes(engine, hj, orc, n):
    p = plan_of(hj, n)
    want = orc.run(orc.port(), p)
    r = engine.execute_raw(p)
    later = engine.execute_raw(plan_of(hj, n, seed=1))
    try:
        check(hj, orc, engine, r, want, 4)
    finally:
        engine.free_result(later)
        engine.free_result(r)


def test_many_results(engine, hj, orc):
    plans = [plan_of(hj, 500 + 7 * k, seed=k) for k in range(20)]
    want = [orc.run(orc.port(), p) for p in plans]
    for _ in range(2):  # the buffers come back
        rs = [engine.execute_raw(p) for p in plans]
        for k in (19, 0, 7, 8, 9, 13):
            check(hj, orc, engine, rs[k], want[k], 4)
        for r in rs:
            engine.free_result(r)


def test_many_columns(engine, hj, orc):
    p = plan_of(hj, 5 * 1984, cols=60)
    r = engine.execute_raw(p)
    try:
        check(hj, orc, engine, r, orc.run(orc.port(), p), 61, ("pages", "pinned"))
    finally:
        engine.free_result(r)


def test_threads(hj, orc):
    """A context each, and results freed by another thread than theirs."""
    failed, done = [], []

    def work(k):
        try:
            e = hj.Engine(0)
            for i in range(10):
                p = plan_of(hj, 100 + 50 * k + i, seed=100 * k + i)
                r = e.execute_raw(p)
                check(hj, orc, e, r, orc.run(orc.port(), p), 4, ("pinned",))
                done.append((e, r))
        except BaseException as x:  # noqa: BLE001
            failed.append(x)

    ts = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for e, r in done:
        e.free_result(r)
    assert not failed, failed
