"""Matches beyond 2^32: counted exactly, with nothing written, by the calls that
only count, and refused by the calls that would have to write them."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb", [5000, 20_000, 70_000])  # a length within its summary's field, and beyond it
@pytest.mark.parametrize("fn", ["hj_table_probe", "hj_table_probe_noalloc"])
def test_more_than_2_32_matches_are_counted(engine, hj, nb, fn):
    """Every probe row is a hit that is listed, at a column length whose list fills its
    memory but for a few entries, and the matches pass 2^32 several times."""
    import torch
    L = hj.lib()
    n = (1 << 20) - 4 if fn == "hj_table_probe" else hj.NOALLOC_MAX_PROBE_ROWS
    keys = torch.full((nb,), 7, dtype=torch.int32, device="cuda")
    probe = torch.full((n,), 7, dtype=torch.int32, device="cuda")
    few = torch.arange(5, 10, dtype=torch.int32, device="cuda")
    out = torch.full((2, nb), -1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    nm, t = C.c_uint64(), C.c_void_p()
    assert L.hj_table_build(engine.handle, keys.data_ptr(), None, nb, -1, C.byref(t)) == 0
    try:
        for _ in range(2):
            assert getattr(L, fn)(engine.handle, t, probe.data_ptr(), None, n, None, None, 0,
                                  C.byref(nm)) == hj.HJ_ERR_CAPACITY
            assert nm.value == n * nb
        assert getattr(L, fn)(engine.handle, t, few.data_ptr(), None, 5, out[0].data_ptr(), out[1].data_ptr(), nb,
                              C.byref(nm)) == 0
        assert nm.value == nb and bool((out[0] == 2).all())
        assert np.array_equal(np.sort(out[1].cpu().numpy()), np.arange(nb))
    finally:
        L.hj_table_free(t)


def test_more_than_2_32_rows_are_not_written(engine, hj):
    """Refused however the matches divide into single ones of their probe row and listed
    ones (here just under 2^32 of these), with buffers that would hold them all."""
    import torch
    L = hj.lib()
    if torch.cuda.mem_get_info()[0] < 60 << 30:
        pytest.skip("needs 60 GB of free device memory")
    heavy, hits, singles = 1 << 16, (1 << 16) - 1, 1 << 17
    keys = torch.full((heavy + 1,), 7, dtype=torch.int32, device="cuda")
    keys[heavy] = 8
    probe = torch.cat([torch.full((hits,), 7), torch.full((singles,), 8)]).int().cuda()
    rows = heavy * hits + singles
    assert heavy * hits < 1 << 32 < rows
    out = [torch.empty(rows, dtype=torch.int32, device="cuda") for _ in range(2)]
    for o in out:
        o[:1000] = -1
    torch.cuda.synchronize()
    nm, t = C.c_uint64(), C.c_void_p()
    assert L.hj_table_build(engine.handle, keys.data_ptr(), None, heavy + 1, -1, C.byref(t)) == 0
    try:
        assert L.hj_table_probe(engine.handle, t, probe.data_ptr(), None, probe.numel(), out[0].data_ptr(),
                                out[1].data_ptr(), rows, C.byref(nm)) == hj.HJ_ERR_INVALID
        assert nm.value == rows and all(int(o[:1000].max()) == -1 for o in out)
    finally:
        L.hj_table_free(t)
