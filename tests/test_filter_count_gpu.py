"""Filtered scans around a tile's size and around the number of tiles up to which
the filter's last block makes their offsets: every passing row, in order, and
the same again (the counter is clear)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 4095, 4096, 4097, 16 * 4096 * 256 + 1, (1 << 14) * 4096, (1 << 14) * 4096 + 1])
@pytest.mark.parametrize("keep", ["none", "all", "some"])
def test_rows_in_order(engine, hj, n, keep):
    v = (np.arange(n, dtype=np.int64) * 2654435761 % 1000).astype(np.int32)
    lit = {"none": 0, "all": 1000, "some": 10}[keep]
    p = hj.Plan()
    p.new_input(hj.Table(n, [hj.Column.int32(v), hj.Column.int32(np.arange(n, dtype=np.int32))]))
    if keep == "all" and n > 1 << 25:
        lit = 990
    p.root = p.new_scan_node(0, [(1, hj.INT32)], [(0, hj.CMP_LT, lit)])
    t = engine.upload(p.inputs[0])
    try:
        q = hj.Plan(p.nodes, [t], p.root)
        for _ in range(2):
            res = engine.execute(q)
            assert np.array_equal(hj.decode_int32(res.columns[0])[0], np.nonzero(v < lit)[0])
    finally:
        engine.release(t)
