"""A request's memory estimate covers the arrays of a join whose sizes follow from its
probe side: the lists, and the output streams made before the matches are counted."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("probe", [100_000, 3_000_000, 30_000_000])
def test_estimate_covers_lists_and_streams(engine, hj, probe):
    I, p = hj.INT32, hj.Plan()
    keys = np.full(probe, -1, np.int32)
    keys[:10] = np.arange(10)
    held = [engine.upload(hj.Table(k.size, [hj.Column.int32(k)] * 2)) for k in (np.arange(1000, dtype=np.int32), keys)]
    for t in held:
        p.new_input(t)
    p.root = p.new_join_node(True, p.new_scan_node(0, [(0, I), (1, I)]), p.new_scan_node(1, [(0, I), (1, I)]), 0, 0,
                             [(0, I), (1, I), (2, I), (3, I)])
    try:
        with engine.server(1 << 40, 1) as srv:
            res, st = srv.wait(srv.submit(p))
            assert engine.stats(res)[2] == 10
            engine.free_result(res)
        # nine words a probe row; a row id of each side for four matches a row, at most 2^24 more
        # than the rows; and, as for any plan, pages for as many rows as the probe side has
        assert st["est_bytes"] >= 36 * probe + 2 * 4 * (probe + min(3 * probe, 1 << 24)) + 4 * 12 * probe
    finally:
        for t in held:
            engine.release(t)
