"""Output columns that share launches: one more than a launch takes of each type,
more VARCHAR ones than the host's scratch has counts, in mixed order, with row counts around a page's and a packing tile's, NULLs,
long strings, and empty results."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def strings(hj, r, n, longest):
    lens = r.integers(0, longest + 1, n)
    if longest > 1000:  # a few long-string pages, the rest short
        lens = np.where(r.random(n) < 0.002, lens, lens % 30)
    offs = np.zeros(n + 1, np.uint64)
    np.cumsum(lens, out=offs[1:])
    data = r.integers(33, 127, max(1, int(offs[-1]))).astype(np.uint8)
    return hj.Column.varchar(data, offs, (r.random(n) < 0.9).astype(np.uint8))


@pytest.mark.parametrize("ints,strs", [(1, 0), (0, 1), (16, 8), (17, 9), (33, 17), (0, 9), (17, 0), (2, 64), (2, 65),
                                       (0, 130)])
@pytest.mark.parametrize("n", [1, 1983, 1985, 4096, 4097, 20_011])
def test_columns(engine, hj, orc, ints, strs, n):
    import test_gpu_parity as tp
    r = np.random.default_rng(ints * 1000 + strs + n)
    cols = [hj.Column.int32(r.permutation(n).astype(np.int32))]
    types = [hj.INT32]
    for k in range(ints):
        valid = (r.random(n) < 0.8).astype(np.uint8) if k % 2 else None
        cols.append(hj.Column.int32(r.integers(-2**31, 2**31, n).astype(np.int32), valid))
        types.append(hj.INT32)
    for k in range(strs):
        cols.append(strings(hj, r, n, 20_000 if k == 3 else 40 * (k % 3)))
        types.append(hj.VARCHAR)
    p = hj.Plan()
    p.new_input(hj.Table(n, cols))
    p.new_input(hj.Table(n, [hj.Column.int32(r.integers(0, n, n).astype(np.int32))]))
    p.new_scan_node(0, list(enumerate(types)))
    p.new_scan_node(1, [(0, hj.INT32)])
    out = r.permutation(np.arange(1, len(types)))
    p.root = p.new_join_node(True, 0, 1, 0, 0, [(int(j), types[j]) for j in out])
    tp.assert_same(orc, engine.execute(p), orc.run(orc.port(), p), f"{ints} {strs} {n}")
