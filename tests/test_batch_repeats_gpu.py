"""The batch where keys repeat (hj_batch_execute, persistent mode): keys with so many
rows in R1 that they are listed beside the table, around the number of rows that
makes a key one of those; keys that later relations hold more than once; results of
a row enumerated by one lane and by a warp.  No instance needs the plain path; row
counts and checksums are equal to the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

import batch_oracle as bo
from test_batch_tables_gpu import FREE, I32, rel, run

pytestmark = pytest.mark.gpu


def check(engine, host, **opts):
    got, redo = run(engine, host, **opts)
    assert got == [bo.chain_result(i) for i in host] and redo == 0


@pytest.mark.parametrize("opts", [{}, {"batch_load_pct": 80}, {"batch_load_pct": 25}, {"batch_part_log2": 8},
                                  {"batch_part_log2": 13}])
def test_hot_keys_in_r1(engine, opts):
    """One key, and several, with 1 to some thousand rows among unique ones; probe rows
    that miss, and some that meet the hot keys."""
    r = np.random.default_rng(1)
    host = []
    top = 300 if opts.get("batch_part_log2") == 8 else 8000
    for hot in (1, 4, 5, 11, 12, 13, 14, 40, 300, 490, 3000, 8000):
        if hot > top:
            continue
        for keys in (1, 3):
            cold = r.choice(np.arange(*I32, 65_537, dtype=np.int64), 2000, replace=False)
            hots = np.array([7, -9, int(FREE)])[:keys]
            k1 = r.permutation(np.concatenate([np.repeat(hots, min(hot, top // keys)), cold[:100 if hot > 1000 else 1000]]))
            probe = np.concatenate([r.choice(cold, 5000), hots, hots[:1], r.integers(*I32, 500)])
            host.append([rel(r, r.permutation(probe)), rel(r, k1)])
    check(engine, host, **opts)


@pytest.mark.parametrize("dup", [2, 3, 7, 8, 9, 12, 13, 16, 33, 100])
@pytest.mark.parametrize("nb", [600, 5000, 30_000])
def test_every_key_repeats(engine, dup, nb):
    r = np.random.default_rng(dup * nb)
    host = []
    for m in (2, 3):
        dom = r.choice(np.arange(*I32, 4001, dtype=np.int64), max(2, nb // dup), replace=False)
        rest = [rel(r, r.permutation(dom)) for _ in range(m - 2)]
        host.append([rel(r, np.concatenate([r.choice(dom, 800), r.integers(*I32, 3000)])),
                     rel(r, r.permutation(np.repeat(dom, dup))), *rest])
        host.append([host[-1][0], rel(r, r.permutation(dom)), *rest, rel(r, r.permutation(np.repeat(dom, dup)))])
    check(engine, host)


@pytest.mark.parametrize("m", range(2, 9))
def test_some_keys_repeat(engine, m):
    """Partitions with and without listed keys in one instance, a different relation with
    the repeated ones each time, and all of them with some."""
    r = np.random.default_rng(m)
    host = []
    for where in list(range(1, m)) + [0]:
        dom = r.choice(np.arange(*I32, 40_009, dtype=np.int64), 20_000, replace=False)
        inst = [rel(r, np.concatenate([r.choice(dom, 20_000), r.integers(*I32, 20_000)]))]
        some = r.choice(dom, 30, replace=False)
        for j in range(1, m):
            k = r.choice(dom, 18_000, replace=False)
            if where in (0, j):
                k = np.concatenate([k, np.repeat(some, 1 if where == 0 and m > 4 else 20 // m), r.choice(k, 5)])
            inst.append(rel(r, r.permutation(k)))
        host.append(inst)
    check(engine, host)


def test_one_key_in_every_relation(engine):
    """A key's combinations: 1 to 9 (a lane's) and tens of thousands (a warp's) a probe row."""
    r = np.random.default_rng(5)
    host = []
    for counts in ((1, 2), (2, 2), (2, 4), (3, 3), (9, 1), (31, 33), (64, 40, 5), (2, 2, 2, 2, 2, 2, 2), (300, 1, 70)):
        other = np.arange(1000, 3000)
        inst = [rel(r, np.concatenate([np.full(5, 7), r.choice(other, 300), np.arange(5000, 9000)]))]
        for c in counts:
            inst.append(rel(r, r.permutation(np.concatenate([np.full(c, 7), other]))))
        host.append(inst)
    check(engine, host)
