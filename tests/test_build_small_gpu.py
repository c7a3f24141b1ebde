"""Table builds of at most 2^16 keys (one launch, every block reading all keys)
and just above: partition and block edges, directories of few and of many bits,
heavy keys beyond the listed tuples, NULL keys.  The directory is UnchainedHash's
where it sizes it, and the probe's matches are those of the keys compared."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class _Dev:
    def __init__(self, ptr, n, typestr):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (ptr, False), "version": 3}


def keys_of(kind, n, r):
    if kind == "perm":
        return r.permutation(n).astype(np.int32)
    if kind == "random":
        return r.integers(-2**31, 2**31, n).astype(np.int32)
    if kind == "dup":
        return r.integers(0, max(1, n // 4), n).astype(np.int32)
    if kind == "half":
        return np.where(r.random(n) < 0.5, -7, r.integers(0, 2**30, n)).astype(np.int32)
    return np.full(n, 2**31 - 1, np.int32)


def check(engine, hj, orc, keys, dir_bits, r, valid=None):
    import torch
    L = hj.lib()
    kb = torch.from_numpy(keys).cuda()
    vb = None
    if valid is not None:
        bits = np.packbits(valid.astype(np.uint8), bitorder="little")
        vb = torch.from_numpy(np.pad(bits, (0, (-bits.size) % 4)).view(np.int32).copy()).cuda()
    t = C.c_void_p()
    assert L.hj_table_build(engine.handle, kb.data_ptr(), None if vb is None else vb.data_ptr(), keys.size, dir_bits,
                            C.byref(t)) == 0
    used = keys if valid is None else keys[valid]
    try:
        bits, nt, d = C.c_uint32(), C.c_uint64(), C.c_void_p()
        tk, tr = C.c_void_p(), C.c_void_p()
        L.hj_table_info(t, C.byref(bits), C.byref(nt), C.byref(d), C.byref(tk), C.byref(tr))
        assert nt.value == used.size
        dev = torch.as_tensor(_Dev(d.value, (1 << bits.value) + 1, "<u8"), device="cuda").cpu().numpy()
        if dir_bits < 0:
            assert np.array_equal(dev.astype(np.uint64), orc.unchained_directory(used).astype(np.uint64))
        rows = torch.as_tensor(_Dev(tr.value, used.size, "<u4"), device="cuda").cpu().numpy().astype(np.int64)
        got = torch.as_tensor(_Dev(tk.value, used.size, "<i4"), device="cuda").cpu().numpy()
        assert np.array_equal(np.sort(rows), np.arange(keys.size) if valid is None else np.flatnonzero(valid))
        assert np.array_equal(keys[rows], got)
        probe = np.concatenate([r.permutation(np.unique(used))[:3000], r.integers(-2**31, 2**31, 500)]).astype(np.int32)
        want = orc.unchained_counts(used, probe)
        kp = torch.from_numpy(probe).cuda()
        cap = int(want.sum())
        op = torch.empty(max(cap, 1), dtype=torch.int32, device="cuda")
        ob = torch.empty(max(cap, 1), dtype=torch.int32, device="cuda")
        nm = C.c_uint64()
        assert L.hj_table_probe(engine.handle, t, kp.data_ptr(), None, kp.numel(), op.data_ptr(), ob.data_ptr(), cap,
                                C.byref(nm)) == 0
        assert nm.value == cap
        pr, br = op[:cap].cpu().numpy(), ob[:cap].cpu().numpy()
        assert np.array_equal(probe[pr], keys[br])
        assert np.array_equal(np.bincount(pr, minlength=probe.size), want)
        assert np.unique(pr.astype(np.int64) << 32 | br).size == cap
    finally:
        L.hj_table_free(t)


@pytest.mark.parametrize("kind", ["perm", "random", "dup", "half", "const"])
@pytest.mark.parametrize("n", [1, 2, 31, 33, 2048, 2049, 20_480, 20_481, 65_535, 65_536, 65_537])
def test_sizes_and_skew(engine, hj, orc, kind, n):
    r = np.random.default_rng(n)
    check(engine, hj, orc, keys_of(kind, n, r), -1, r)


@pytest.mark.parametrize("dir_bits", [0, 1, 4, 5, 6, 12, 13, 14, 18, 20])
@pytest.mark.parametrize("n", [3, 5000, 60_000])
def test_directory_bits(engine, hj, orc, dir_bits, n):
    r = np.random.default_rng(dir_bits * 7 + n)
    check(engine, hj, orc, keys_of("dup", n, r), dir_bits, r)


@pytest.mark.parametrize("n", [40, 5000, 65_536])
def test_null_keys(engine, hj, orc, n):
    r = np.random.default_rng(n)
    check(engine, hj, orc, keys_of("dup", n, r), -1, r, valid=r.random(n) < 0.8)


@pytest.mark.parametrize("n", [700, 9000, 50_000])
def test_column_with_nulls_through_execute(engine, hj, orc, n):
    """A build column with NULLs read as value_t, its non-NULL count known from the page headers."""
    import test_gpu_parity as tp
    r = np.random.default_rng(n)
    k, v = r.integers(0, n, n).astype(np.int32), (r.random(n) < 0.9).astype(np.uint8)
    p = hj.Plan()
    p.new_input(hj.Table(n, [hj.Column.int32(k, v), hj.Column.int32(np.arange(n, dtype=np.int32))]))
    p.new_input(hj.Table(3000, [hj.Column.int32(r.integers(0, n, 3000).astype(np.int32))]))
    p.new_scan_node(0, [(0, hj.INT32), (1, hj.INT32)])
    p.new_scan_node(1, [(0, hj.INT32)])
    p.root = p.new_join_node(True, 0, 1, 0, 0, [(0, hj.INT32), (1, hj.INT32), (2, hj.INT32)])
    tp.assert_same(orc, engine.execute(p), orc.run(orc.port(), p), "nulls")
