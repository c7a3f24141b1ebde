"""Input columns that are decoded in one launch: more than a launch takes, each
kind after each other one, pages around the warps of a block, long strings, an
empty table; prepared tables and raw ones give the same rows."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def column(hj, r, kind, n):
    v = r.integers(-2**31, 2**31, n).astype(np.int32)
    if kind == "dense":
        return hj.Column.int32(v), hj.INT32
    if kind == "nulls":
        return hj.Column.int32(v, (r.random(n) < 0.7).astype(np.uint8)), hj.INT32
    if kind == "all_null":
        return hj.Column.int32(v, np.zeros(n, np.uint8)), hj.INT32
    lens = r.integers(0, 40, n)
    if kind == "long" and n:
        lens[r.integers(0, n, 2)] = 20_000
    offs = np.zeros(n + 1, np.uint64)
    np.cumsum(lens, out=offs[1:])
    data = r.integers(33, 127, max(1, int(offs[-1]))).astype(np.uint8)
    return hj.Column.varchar(data, offs, (r.random(n) < 0.9).astype(np.uint8)), hj.VARCHAR


@pytest.mark.parametrize("n", [0, 1, 1984, 1985, 15_872, 15_873, 40_000])
@pytest.mark.parametrize("prepared", [False, True])
def test_columns(engine, hj, orc, n, prepared):
    import test_gpu_parity as tp
    r = np.random.default_rng(n)
    kinds = ["nulls", "text", "dense", "long", "all_null", "nulls", "long"]
    p, types = hj.Plan(), []
    for t in range(3):  # 21 columns to decode or read in place, over three scans
        cols = [(hj.Column.int32(r.permutation(n).astype(np.int32)), hj.INT32)]
        cols += [column(hj, r, k, n) for k in (kinds[t:] + kinds[:t])]
        p.new_input(hj.Table(n, [c for c, _ in cols]))
        types.append([ty for _, ty in cols])
        p.new_scan_node(t, list(enumerate(types[t])))
    two = types[0] + types[1]
    a = p.new_join_node(True, 0, 1, 0, 0, list(enumerate(two)))
    p.root = p.new_join_node(False, a, 2, 0, 0, list(enumerate(two + types[2])))
    want = orc.run(orc.port(), p)
    if not prepared:
        tp.assert_same(orc, engine.execute(p), want, str(n))
        return
    res = [engine.upload(t) for t in p.inputs]
    try:
        for t in res:
            engine.prepare(t)
        q = hj.Plan(p.nodes, res, p.root)
        for _ in range(2):
            tp.assert_same(orc, engine.execute(q), want, f"prepared {n}")
    finally:
        for t in res:
            engine.release(t)
