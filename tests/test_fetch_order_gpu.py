"""Fetching a result column is ordered after the work that the program has put on
the engine's stream, whatever the column's pages: a read of the destination that
is still to run gets what was there before."""
from __future__ import annotations

import ctypes as C

import pytest

from test_result_fetch_gpu import plan_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [50, 10_000, 40_000])  # 1, 6 and 21 pages
@pytest.mark.parametrize("how", ["contiguous", "pages"])
def test_reads_of_the_buffer_come_first(engine, hj, rows, how):
    import torch
    L = hj.lib()
    res = engine.execute_raw(plan_of(hj, rows, cols=1, strings=False))
    try:
        n = C.c_uint64()
        assert L.hj_result_column(res, 0, None, C.byref(n)) == 0
        buf = torch.full((int(n.value), hj.PAGE_SIZE), 0xA5, dtype=torch.uint8).pin_memory()
        seen = torch.zeros_like(buf, device="cuda")
        torch.cuda.synchronize()
        with torch.cuda.stream(torch.cuda.ExternalStream(engine.stream)):
            torch.cuda._sleep(40_000_000)  # some 20 ms
            seen.copy_(buf, non_blocking=True)
        if how == "pages":
            ptrs = (C.c_void_p * int(n.value))(*[buf[i].data_ptr() for i in range(int(n.value))])
            assert L.hj_result_copy_pages(engine.handle, res, 0, ptrs) == 0
        else:
            assert L.hj_result_copy_contiguous(engine.handle, res, 0, buf.data_ptr()) == 0
        torch.cuda.synchronize()
        assert bool((seen == 0xA5).all())
        assert int(buf[0, 0]) | int(buf[0, 1]) << 8 == min(rows, 1984)  # and the pages are there
    finally:
        engine.free_result(res)
