"""The probe's count kernels where they can go wrong: columns of one tile of rows
(a block in order) and of several (warps with queues), around the tile's, a
step's and a queue's sizes, against tables of single tuples, duplicates, small
and large mixed buckets, and a bucket longer than its summary can say; every
match once.  With NULL keys, without outputs, and allocation-free."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def build_keys(kind, r):
    if kind == "unique":
        return r.permutation(5000).astype(np.int32)
    if kind == "pairs":
        return r.permutation(np.repeat(np.arange(3000), 2)).astype(np.int32)
    if kind == "some":  # mostly unique, a few keys several times
        return np.concatenate([r.permutation(5000), r.integers(0, 5000, 300)]).astype(np.int32)
    return np.concatenate([np.full(40_000, 17), r.permutation(3000)]).astype(np.int32)  # heavy


@pytest.mark.parametrize("n", [1, 31, 33, 1983, 1984, 1985, 2047, 3968, 3969, 40_001])
@pytest.mark.parametrize("kind,dir_bits", [("unique", -1), ("unique", 9), ("unique", 5), ("unique", 0), ("pairs", -1),
                                           ("pairs", 8), ("some", -1), ("some", 12), ("heavy", -1), ("heavy", 6)])
def test_matches(engine, hj, n, kind, dir_bits):
    import torch
    L = hj.lib()
    r = np.random.default_rng(n * 31 + dir_bits)
    keys = build_keys(kind, r)
    probe = r.integers(-50, 5600, n).astype(np.int32)
    if kind == "heavy":
        probe[:] = np.where(probe == 17, 18, probe)
        probe[: min(n, 3)] = 17
    valid = r.random(n) < 0.9
    bits = np.packbits(valid.astype(np.uint8), bitorder="little")
    vb = torch.from_numpy(np.pad(bits, (0, (-bits.size) % 4)).view(np.int32).copy()).cuda()
    kb, kp = torch.from_numpy(keys).cuda(), torch.from_numpy(probe).cuda()
    order = np.argsort(keys, kind="stable")
    lo, hi = np.searchsorted(keys[order], probe, "left"), np.searchsorted(keys[order], probe, "right")
    t = C.c_void_p()
    assert L.hj_table_build(engine.handle, kb.data_ptr(), None, keys.size, dir_bits, C.byref(t)) == 0
    try:
        for v in (None, valid):
            cnt = hi - lo if v is None else np.where(v, hi - lo, 0)
            prow = np.repeat(np.arange(n), cnt)
            at = np.repeat(lo, cnt) + np.arange(prow.size) - np.repeat(np.cumsum(cnt) - cnt, cnt)
            want = np.sort(prow.astype(np.int64) << 32 | order[at])
            cap = int(want.size)
            nm = C.c_uint64()
            vp = None if v is None else vb.data_ptr()
            if cap:  # the count alone
                assert L.hj_table_probe(engine.handle, t, kp.data_ptr(), vp, n, None, None, 0,
                                        C.byref(nm)) == hj.HJ_ERR_CAPACITY
                assert nm.value == cap
            for fn in (L.hj_table_probe, L.hj_table_probe_noalloc):
                op = torch.full((cap + 1,), -1, dtype=torch.int32, device="cuda")
                ob = torch.full((cap + 1,), -1, dtype=torch.int32, device="cuda")
                if cap > 1:  # one slot short: the count, and nothing written
                    assert fn(engine.handle, t, kp.data_ptr(), vp, n, op.data_ptr(), ob.data_ptr(), cap - 1,
                              C.byref(nm)) == hj.HJ_ERR_CAPACITY
                    assert nm.value == cap and int(op.max()) == -1 and int(ob.max()) == -1
                assert fn(engine.handle, t, kp.data_ptr(), vp, n, op.data_ptr(), ob.data_ptr(), cap, C.byref(nm)) == 0
                assert nm.value == cap and int(op[cap]) == -1 and int(ob[cap]) == -1
                got = op[:cap].cpu().numpy().astype(np.int64) << 32 | ob[:cap].cpu().numpy()
                assert np.array_equal(np.sort(got), want)
    finally:
        L.hj_table_free(t)


@pytest.mark.parametrize("opts", [{"light_max": 1}, {"light_max": 31}, {"light_max": 32}, {"light_max": 1000}])
@pytest.mark.parametrize("n", [1500, 30_000])
def test_light_max(engine, hj, orc, n, opts):
    """Few buckets of many keys: compared by a lane, or listed for a warp or block each."""
    import test_gpu_parity as tp
    r = np.random.default_rng(n)
    p = hj.Plan()
    p.new_input(hj.Table(4000, [hj.Column.int32(r.integers(0, 3000, 4000).astype(np.int32)),
                                hj.Column.int32(np.arange(4000, dtype=np.int32))]))
    p.new_input(hj.Table(n, [hj.Column.int32(r.integers(0, 4000, n).astype(np.int32)),
                             hj.Column.int32(np.arange(n, dtype=np.int32))]))
    p.new_scan_node(0, [(0, hj.INT32), (1, hj.INT32)])
    p.new_scan_node(1, [(0, hj.INT32), (1, hj.INT32)])
    p.root = p.new_join_node(True, 0, 1, 0, 0, [(1, hj.INT32), (3, hj.INT32)])
    want = orc.run(orc.port(), p)
    opts = dict(opts, dir_bits=7)
    saved = {k: engine.get_option(k) for k in opts}
    try:
        for k, v in opts.items():
            engine.set_option(k, v)
        tp.assert_same(orc, engine.execute(p), want, str(opts))
        tp.assert_same(orc, engine.execute(p), want, str(opts))  # the counters are clear again
    finally:
        for k, v in saved.items():
            engine.set_option(k, v)
