"""The match writer where its output streams do not start on a 16-byte boundary: behind
0 to 5 directly written rows, and in buffers of the caller at any word (both alike,
or each at its own), with results around its chunks' sizes, and one hit over several
chunks; every option of rows a thread.  Nothing beside the result is written."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("group", [1, 2, 4, 8, 16])
@pytest.mark.parametrize("direct", range(6))
def test_every_alignment(engine, hj, group, direct):
    import torch
    L = hj.lib()
    r = np.random.default_rng(group * 7 + direct)
    saved = engine.get_option("probe_group")
    engine.set_option("probe_group", group)
    chunk = 32 * group
    try:
        for dup, hits in ((2, 1), (2, chunk // 2), (3, (2 * chunk + 1) // 3), (chunk - 1, 1), (chunk, 1), (chunk + 1, 2),
                          (5, chunk + 1), (3 * chunk + 2, 2), (7, 3000)):
            # the keys of listed hits `dup` times, those of single matches once
            heavy = np.arange(100, 100 + min(hits, 600))
            build = r.permutation(np.concatenate([np.repeat(heavy, dup), np.arange(direct)])).astype(np.int32)
            probe = np.concatenate([np.resize(heavy, hits), np.arange(direct), np.full(3000, -7)]).astype(np.int32)
            probe = r.permutation(probe)
            order = np.argsort(build, kind="stable")
            lo, hi = np.searchsorted(build[order], probe, "left"), np.searchsorted(build[order], probe, "right")
            cnt = hi - lo
            prow = np.repeat(np.arange(probe.size), cnt)
            at = np.repeat(lo, cnt) + np.arange(prow.size) - np.repeat(np.cumsum(cnt) - cnt, cnt)
            want = np.sort(prow.astype(np.int64) << 32 | order[at])
            kb, kp = torch.from_numpy(build).cuda(), torch.from_numpy(probe).cuda()
            t, nm = C.c_void_p(), C.c_uint64()
            torch.cuda.synchronize()
            assert L.hj_table_build(engine.handle, kb.data_ptr(), None, build.size, -1, C.byref(t)) == 0
            try:
                for fn in (L.hj_table_probe, L.hj_table_probe_noalloc):
                    for a, b in ((0, 0), (1, 1), (2, 2), (3, 3), (0, 2), (3, 1)):
                        out = torch.full((2, want.size + 16), -1, dtype=torch.int32, device="cuda")
                        torch.cuda.synchronize()
                        assert fn(engine.handle, t, kp.data_ptr(), None, probe.size, out[0, 4 + a:].data_ptr(),
                                  out[1, 4 + b:].data_ptr(), want.size, C.byref(nm)) == 0
                        o = out.cpu().numpy()
                        got = o[0, 4 + a:4 + a + want.size].astype(np.int64) << 32 | o[1, 4 + b:4 + b + want.size]
                        assert nm.value == want.size and np.array_equal(np.sort(got), want)
                        assert (o == -1).sum() == 32
            finally:
                L.hj_table_free(t)
    finally:
        engine.set_option("probe_group", saved)


@pytest.mark.parametrize("direct", range(5))
def test_join_streams_behind_direct_rows(engine, hj, orc, direct):
    """A join with three sources, two of them read through row ids."""
    import test_gpu_parity as tp
    r = np.random.default_rng(direct)
    I, p = hj.INT32, hj.Plan()
    n = 40_000
    fk = r.integers(1000, 3000, n).astype(np.int32)
    fk[:direct] = np.arange(direct)
    dim = np.concatenate([np.repeat(np.arange(1000, 3000), 3), np.arange(10)]).astype(np.int32)
    for cols in ([r.permutation(dim), np.arange(dim.size)], [fk, np.arange(n)], [np.arange(n), r.integers(0, 9, n)]):
        p.new_input(hj.Table(len(cols[0]), [hj.Column.int32(np.asarray(c, np.int32)) for c in cols]))
    s = [p.new_scan_node(i, [(0, I), (1, I)]) for i in range(3)]
    mid = p.new_join_node(False, s[1], s[2], 1, 0, [(0, I), (1, I), (3, I)])
    p.root = p.new_join_node(True, s[0], mid, 0, 0, [(1, I), (3, I), (4, I), (0, I)])
    tp.assert_same(orc, engine.execute(p), orc.run(orc.port(), p), str(direct))
