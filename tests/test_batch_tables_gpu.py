"""The batch's hash tables (hj_batch_execute, persistent mode) where they can go
wrong: relation sizes at the edges of buckets, blocks and work items, chains of
2 to 8 relations with and without duplicate keys, runs of equal rows through
many buckets, long partner lists, and rows equal to the pattern of a free slot.
Row counts and checksums are whole numbers: equal to the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

import batch_oracle as bo

pytestmark = pytest.mark.gpu

FREE = np.uint32(0x81818181).astype(np.int32)  # key and payload of a free slot
I32 = (-2**31, 2**31)


def run(engine, host, **opts):
    import torch
    keep, insts = [], []
    for inst in host:
        rels = []
        for k, v in inst:
            tk = torch.from_numpy(np.ascontiguousarray(k, np.int32)).cuda()
            tv = torch.from_numpy(np.ascontiguousarray(v, np.int32)).cuda()
            keep += [tk, tv]
            rels.append((tk.data_ptr(), tv.data_ptr(), tk.numel()))
        insts.append(rels)
    torch.cuda.synchronize()
    saved = {o: engine.get_option(o) for o in opts}
    try:
        for o, v in opts.items():
            engine.set_option(o, v)
        rows, sums, redo = engine.batch_execute(insts)
    finally:
        for o, v in saved.items():
            engine.set_option(o, v)
    return [(int(a), int(b)) for a, b in zip(rows, sums)], redo


def rel(r, keys):
    keys = np.asarray(keys, np.int32)
    return keys, r.integers(*I32, keys.size).astype(np.int32)


@pytest.mark.parametrize("nb", [1, 2, 4, 5, 511, 4096, 4097, 8192, 8193, 70_001])
@pytest.mark.parametrize("n0", [1, 511, 513, 8191, 8193, 70_001])
def test_sizes(engine, nb, n0):
    r = np.random.default_rng(nb * 100_003 + n0)
    host = []
    for m in (2, 3, 5):
        dom = r.choice(np.arange(*I32, 4001, dtype=np.int64), 2 * nb, replace=False)
        host.append([rel(r, r.choice(dom, n0))] + [rel(r, r.choice(dom, nb, replace=False)) for _ in range(m - 1)])
    got, redo = run(engine, host)
    assert got == [bo.chain_result(i) for i in host] and redo == 0


@pytest.mark.parametrize("m", range(2, 9))
@pytest.mark.parametrize("opts", [{}, {"batch_part_log2": 9}, {"batch_load_pct": 200}, {"batch_load_pct": 20}])
def test_depths_and_duplicates(engine, m, opts):
    """Keys in arithmetic progression, each relation with its own share of duplicates."""
    r = np.random.default_rng(m)
    dom = np.arange(6000) * 2654435761 % (1 << 32)
    dom = dom.astype(np.uint32).view(np.int32)
    host = []
    for dup in (0, m - 1, 1, m // 2):  # which relation holds duplicates (0: none)
        inst = [rel(r, r.choice(dom, 30_000))]
        for j in range(1, m):
            k = r.choice(dom, 4000, replace=False)
            if j == dup:
                k = np.concatenate([k, r.choice(k, 400), r.choice(k, 50)])
            inst.append(rel(r, r.permutation(k)))
        host.append(inst)
    got, redo = run(engine, host, **opts)
    assert got == [bo.chain_result(i) for i in host] and redo == 0


@pytest.mark.parametrize("m", [2, 3, 4])
def test_equal_rows_and_long_partner_lists(engine, m):
    """One (key, payload) pair many times in every build relation: buckets of
    equal slots, runs over hundreds of buckets, lists longer than a thread keeps."""
    r = np.random.default_rng(m)
    host = []
    for reps in (4, 5, 8, 9, 30, 900 if m == 2 else 60):
        inst = [(np.concatenate([np.full(3, 7), r.integers(0, 500, 2000)]).astype(np.int32),
                 np.zeros(2003, np.int32))]
        for j in range(1, m):
            k = np.concatenate([np.full(reps, 7), r.permutation(np.arange(10, 400))]).astype(np.int32)
            inst.append((k, np.where(k == 7, 5, k).astype(np.int32)))
        host.append(inst)
    got, redo = run(engine, host)
    assert got == [bo.chain_result(i) for i in host] and redo == 0


def test_free_slot_pattern(engine):
    """The key of a free slot joins like any other; a build row that is the whole
    pattern sends its instance to the plain path, with the same result."""
    r = np.random.default_rng(3)
    some = r.integers(*I32, 3000).astype(np.int32)
    probe = rel(r, np.concatenate([some, np.full(40, FREE)]))
    with_key = rel(r, np.concatenate([some[:900], [FREE, FREE]]))
    whole = (np.append(some[:900], FREE).astype(np.int32), np.append(some[:900], FREE).astype(np.int32))
    host = [[probe, with_key], [probe, rel(r, some[:900])], [probe, with_key, with_key], [probe, whole],
            [probe, with_key, whole], [probe, rel(r, some[:900])]]
    got, redo = run(engine, host)
    assert got == [bo.chain_result(i) for i in host]
    assert redo <= 2  # only the instances that hold the pattern


def test_graph_is_updated_between_batches(engine):
    """Batches of other sizes and depths one after another on one context, with and without the graph."""
    r = np.random.default_rng(8)
    for opts in ({}, {"batch_graph": 0}, {}):
        for m, nb in ((2, 3000), (4, 20_000), (2, 100), (3, 50_000), (2, 0), (2, 3000)):
            dom = np.arange(2 * max(nb, 1))
            host = [[rel(r, r.choice(dom, 10 * max(nb, 5)))] + [rel(r, r.permutation(dom)[:nb]) for _ in range(m - 1)]
                    for _ in range(3)]
            got, redo = run(engine, host, **opts)
            assert got == [bo.chain_result(i) for i in host] and redo == 0
