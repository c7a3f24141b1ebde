"""Joins whose build side is first cut down to the rows that a short probe side
can meet: around the sizes where that rule begins and ends, with NULL keys, no
match, keys of many rows on either side, a cut that keeps too much, filters, row
ids from earlier joins, an output of either side alone, and the tile's order."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def place(i):
    """A row's place in its tile's order."""
    return (i // 32 % 8) * 256 + i // 256 * 32 + i % 32


def plan_of(hj, bkeys, pkeys, bvalid=None, pvalid=None, out=(1, 3)):
    p = hj.Plan()
    for k, v in ((bkeys, bvalid), (pkeys, pvalid)):
        ok = None if v is None else v.astype(np.uint8)
        p.new_input(hj.Table(k.size, [hj.Column.int32(k.astype(np.int32), ok),
                                      hj.Column.int32(np.arange(k.size, dtype=np.int32))]))
        p.new_scan_node(len(p.inputs) - 1, [(0, hj.INT32), (1, hj.INT32)])
    p.root = p.new_join_node(True, 0, 1, 0, 0, [(j, hj.INT32) for j in out])
    return p


def check(engine, orc, p, what):
    import test_gpu_parity as tp
    want = orc.run(orc.port(), p)
    for _ in range(2):  # the counters are clear again
        res = engine.execute(p)
        tp.assert_same(orc, res, want, what)
    return res


@pytest.mark.parametrize("nb,n", [(65_536, 100), (65_537, 0), (65_537, 1), (65_537, 4096), (65_537, 4097),
                                  (70_001, 33), (70_001, 1984), (70_001, 1985), (300_001, 8192), (300_001, 8193)])
@pytest.mark.parametrize("kind", ["unique", "heavy_build", "heavy_probe", "none"])
def test_sizes(engine, hj, orc, nb, n, kind):
    r = np.random.default_rng(nb + n)
    b, q = r.permutation(nb), r.integers(0, 2 * nb, n)
    if kind == "heavy_build":  # a heavy key that stays, or one that makes the cut useless
        b[r.permutation(nb)[:17_000 if n % 2 else nb // 2 + 100]] = 5
        q[: min(n, 2)] = 5
    elif kind == "heavy_probe":  # one key of the probe rows many times
        q[r.random(n) < 0.7] = 9
    elif kind == "none":
        q += nb
    check(engine, orc, plan_of(hj, b, q, r.random(nb) < 0.9, r.random(n) < 0.9), f"{kind} {nb} {n}")


@pytest.mark.parametrize("n", [1, 1024, 1984])
def test_order(engine, hj, orc, n):
    """A tile's matches come in its rows' places (keys of three rows each)."""
    r = np.random.default_rng(n)
    b = np.repeat(np.arange(40_000), 3)
    res = check(engine, orc, plan_of(hj, b[r.permutation(b.size)], r.permutation(40_000)[:n]), str(n))
    at = place(np.asarray(hj.decode_int32(res.columns[1])[0], dtype=np.int64))
    assert at.size == 3 * n and np.all(np.diff(at) >= 0)


@pytest.mark.parametrize("out", [(0,), (1,), (2,), (3,), (3, 1, 0, 2)])
def test_outputs(engine, hj, orc, out):
    r = np.random.default_rng(3)
    check(engine, orc, plan_of(hj, r.integers(0, 9000, 90_001), r.integers(0, 9000, 1500), out=out), str(out))


@pytest.mark.parametrize("side", ["build", "probe", "both"])
def test_filters(engine, hj, side):
    r = np.random.default_rng(6)
    p = hj.Plan()
    keys, kept = [], []
    for n, keep in ((150_001, side != "probe"), (4000, side != "build")):
        keys.append(r.integers(0, 40_000, n).astype(np.int32))
        kept.append(3 * n // 4 if keep else n)
        p.new_input(hj.Table(n, [hj.Column.int32(keys[-1]), hj.Column.int32(np.arange(n, dtype=np.int32))]))
        p.new_scan_node(len(p.inputs) - 1, [(0, hj.INT32), (1, hj.INT32)],
                        [(1, hj.CMP_LT, kept[-1])] if keep else [])
    p.root = p.new_join_node(True, 0, 1, 0, 0, [(1, hj.INT32), (3, hj.INT32)])
    res = engine.execute(p)
    i, j = (hj.decode_int32(c)[0].astype(np.int64) for c in res.columns)
    b, q = keys[0][: kept[0]], keys[1][: kept[1]]
    order = np.argsort(b, kind="stable")
    lo, hi = np.searchsorted(b[order], q, "left"), np.searchsorted(b[order], q, "right")
    cnt = hi - lo
    at = np.repeat(lo, cnt) + np.arange(cnt.sum()) - np.repeat(np.cumsum(cnt) - cnt, cnt)
    want = np.sort(np.repeat(np.arange(q.size), cnt) << 32 | order[at])
    assert np.array_equal(np.sort(j << 32 | i), want)


def test_row_ids(engine, hj, orc):
    """Both sides come out of joins: the short one by its row ids, and the large one."""
    r = np.random.default_rng(4)
    i = hj.INT32
    p = hj.Plan()
    for n, dom in ((5000, 5000), (200_000, 5000), (3000, 200_000), (900, 3000)):
        p.new_input(hj.Table(n, [hj.Column.int32(r.permutation(n).astype(np.int32)),
                                 hj.Column.int32(r.integers(0, dom, n).astype(np.int32))]))
        p.new_scan_node(len(p.inputs) - 1, [(0, i), (1, i)])
    a = p.new_join_node(True, 0, 1, 0, 1, [(2, i), (1, i)])     # 200,000 rows
    b = p.new_join_node(True, 2, 3, 0, 1, [(1, i), (2, i)])     # 900 rows
    p.root = p.new_join_node(True, a, b, 0, 0, [(0, i), (1, i), (3, i)])
    check(engine, orc, p, "row ids")
