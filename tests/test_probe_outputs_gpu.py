"""hj_table_probe's pairs in output buffers of any 4-byte alignment, with counts
around what a thread copies at once; nothing beyond them is written."""
from __future__ import annotations

import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 4, 5, 1985, 4096, 16_385, 700_001])
@pytest.mark.parametrize("pa,pb", [(0, 0), (1, 0), (0, 3), (2, 1)])
def test_alignment(engine, hj, n, pa, pb):
    import torch
    L = hj.lib()
    keys = torch.randperm(50_000, device="cuda").int()
    probe = torch.randint(0, 50_000, (n,), device="cuda", dtype=torch.int32)
    a = torch.full((n + 8,), -7, dtype=torch.int32, device="cuda")
    b = torch.full((n + 8,), -7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    t, nm = C.c_void_p(), C.c_uint64()
    assert L.hj_table_build(engine.handle, keys.data_ptr(), None, keys.numel(), -1, C.byref(t)) == 0
    try:
        assert L.hj_table_probe(engine.handle, t, probe.data_ptr(), None, n, a[pa:].data_ptr(), b[pb:].data_ptr(), n,
                                C.byref(nm)) == 0
    finally:
        L.hj_table_free(t)
    assert nm.value == n
    x, y = a[pa:pa + n].long(), b[pb:pb + n].long()
    assert torch.equal(torch.sort(x).values, torch.arange(n, device="cuda"))
    assert torch.equal(keys[y], probe[x])
    for buf, p in ((a, pa), (b, pb)):
        assert bool((buf[:p] == -7).all()) and bool((buf[p + n:] == -7).all())
