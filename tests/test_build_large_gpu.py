"""Builds of several launches: partitions around the size that one block takes,
chunks around their edges, directories of less than a word of mixed bits a
partition, NULL keys, and both sides of the line up to which the heavy
partitions' phases share a launch.  Every build row is found under its key."""
from __future__ import annotations

import ctypes as C

import pytest

pytestmark = pytest.mark.gpu

FUSE, CHUNK, ONE = 12288, 8192, 1 << 22


@pytest.mark.parametrize("n,heavy", [(65_537, 0), (65_537, FUSE), (65_537, FUSE + 1), (70_000, 2 * CHUNK),
                                     (70_000, 2 * CHUNK + 1), (70_000, 69_999), (300_000, 300_000),
                                     (ONE, ONE // 2), (ONE + 1, ONE // 2), (ONE + 1, 0), (ONE + 1, ONE + 1)])
@pytest.mark.parametrize("dir_bits", [-1, 3, 14])
@pytest.mark.parametrize("nulls", [False, True])
def test_rows(engine, hj, n, heavy, dir_bits, nulls):
    import torch
    if n > 1_000_000 and dir_bits == 3:
        pytest.skip("a bucket of half a million keys")
    L = hj.lib()
    g = torch.Generator(device="cuda")
    g.manual_seed(n + heavy)
    keys = torch.randperm(n, generator=g, device="cuda").int()
    keys[torch.randperm(n, generator=g, device="cuda")[:heavy]] = -5
    ok = torch.ones(n, dtype=torch.bool, device="cuda")
    vp = None
    if nulls:
        words = torch.randint(-2**31, 2**31, ((n + 31) // 32,), generator=g, device="cuda").int()
        i = torch.arange(n, device="cuda")
        ok = (words[i // 32] >> (i % 32).int()) & 1 == 1
        vp = words.data_ptr()
    torch.cuda.synchronize()
    want = torch.nonzero(ok).flatten()
    probe = torch.unique(keys[ok])
    probe = torch.cat([probe, probe[-1:] + 1 + torch.arange(100, device="cuda", dtype=torch.int32)])
    cap = want.numel()
    op = torch.full((cap,), -1, dtype=torch.int32, device="cuda")
    ob = torch.full((cap,), -1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    t, nm = C.c_void_p(), C.c_uint64()
    assert L.hj_table_build(engine.handle, keys.data_ptr(), vp, n, dir_bits, C.byref(t)) == 0
    try:
        assert L.hj_table_probe(engine.handle, t, probe.data_ptr(), None, probe.numel(), op.data_ptr(), ob.data_ptr(),
                                cap, C.byref(nm)) == 0
        assert nm.value == cap
        assert torch.equal(torch.sort(ob.long()).values, want)
        assert torch.equal(probe[op.long()], keys[ob.long()])
    finally:
        L.hj_table_free(t)
