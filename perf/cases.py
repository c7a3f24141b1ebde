"""The calls that this engine is timed on, over the range of sizes in which they are used.

Six kinds of work, each through the entry points that a program calls:

  chain   a left-deep chain: a short driving relation meets one dimension table after the
          other (hashed on their unique keys).  The interactive query; latency and launches
          count.
  funnel  a two-join plan: a fact table meets a dimension table, and the large intermediate
          is hashed and met by a short list of selected fact ids.  The analytic query; table
          build and probe count.
  fanout  a short relation with strings against a skewed fact table hashed on its foreign
          key: few probe rows, many result rows; build of heavy keys, match writer and page
          writers count.
  scan    a filtered scan: decode, filter and page writers.
  lookup  the hash-table calls on device columns (hj_table_build / hj_table_probe): for each
          probe row its build row, as a program uses a join as a lookup.
  batch   Engine.batch_execute over many independent join chains, at once or one at a time.

The first four are Engine.execute_raw over resident tables, and the result pages fetched into
page-locked buffers that the program keeps, sized for the most rows that it expects.

The order of a join's result rows is unspecified.  The plans here have outputs that do not
depend on it: the last join's probe side is at most one tile of rows, whose matches come out
in order, and build rows of one key show equal values; a lookup is put in the probe rows'
own order; a batch gives counts and checksums.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from __graft_entry__ import load

hj = load()
from hjgb300 import batch, workloads  # noqa: E402

I, V = hj.INT32, hj.VARCHAR
SHORT = 1984  # rows of a short relation, at most: one tile of the probe
RANK0 = 32    # a fan-out's popular keys start at this rank
_engine = None


def engine() -> "hj.Engine":
    """The program's one engine."""
    global _engine
    if _engine is None:
        _engine = hj.Engine(0)
    return _engine


def listed() -> list:
    return [
        # a point query of a service over tables kept decoded in HBM
        {"name": "chain_point", "kind": "chain", "rels": 2, "rows": 997, "dim_rows": 500, "strings": True,
         "prepared": True},
        # a five-relation chain, as the synthetic chain workload at a small scale; raw pages decoded per call
        {"name": "chain_deep", "kind": "chain", "rels": 5, "rows": 1900, "dim_rows": 120_000, "strings": True,
         "prepared": False},
        # 10M uniform foreign keys over 1M unique keys, the plain 2-table join's shape, then a selection
        {"name": "funnel_uniform", "kind": "funnel", "fact_rows": 10_000_000, "dim_rows": 1_000_000, "dup": 1,
         "skew": 0.0, "sel_rows": 1000, "prepared": False},
        # Zipf foreign keys against a build side with duplicate keys (many-to-many), odd sizes
        {"name": "funnel_skewed", "kind": "funnel", "fact_rows": 3_333_333, "dim_rows": 1_500_001, "dup": 3,
         "skew": 1.1, "sel_rows": 1203, "prepared": True},
        # a build side of Zipf(1.1) keys; 400 of its popular ones fan out to some 0.8M rows with strings
        {"name": "fanout_strings", "kind": "fanout", "fact_rows": 4_000_000, "rows": 400, "strings": True},
        # predicate of 10% selectivity over a raw INT32 table (the raw skewed workload's scan)
        {"name": "scan_large", "kind": "scan", "rows": 16_000_000, "sel": 0.1, "strings": False, "filters": 1},
        # two predicates over a table with strings, a third of the rows kept, odd size
        {"name": "scan_strings", "kind": "scan", "rows": 777_777, "sel": 0.33, "strings": True, "filters": 2},
        # device columns: table built and probed in the pass, 30% misses
        {"name": "lookup_build", "kind": "lookup", "build_rows": 1_000_000, "probe_rows": 10_000_000, "match": 0.7,
         "nulls": False, "kept": False},
        # a table that the program keeps, probed by a smaller column with NULLs
        {"name": "lookup_kept", "kind": "lookup", "build_rows": 262_145, "probe_rows": 1_000_003, "match": 0.9,
         "nulls": True, "kept": True},
        # many small chains at once
        {"name": "batch_small", "kind": "batch", "n": 64, "lo": 1_000, "hi": 16_000, "dup": 1, "plain": False},
        # the batched workload's own mix of sizes, 1k to 4M build rows
        {"name": "batch_mixed", "kind": "batch", "n": 64, "lo": 1_000, "hi": 4_000_000, "dup": 1, "plain": False},
        # one chain at a time through the regular build and probe
        {"name": "batch_plain", "kind": "batch", "n": 6, "lo": 50_000, "hi": 1_000_000, "dup": 1, "plain": True},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(("chain", "funnel", "fanout", "scan", "lookup", "batch", "batch"))
    if kind == "chain":
        return {"kind": kind, "rels": rng.randint(2, 5), "rows": _log_int(rng, 1, SHORT),
                "dim_rows": _log_int(rng, 50, 300_000), "strings": rng.random() < 0.6, "prepared": rng.random() < 0.5}
    if kind == "funnel":
        return {"kind": kind, "fact_rows": _log_int(rng, 5_000, 10_000_000), "dim_rows": _log_int(rng, 500, 2_000_000),
                "dup": rng.choice((1, 1, 3)), "skew": rng.choice((0.0, 1.1)), "sel_rows": rng.randint(1, SHORT),
                "prepared": rng.random() < 0.5}
    if kind == "fanout":
        return {"kind": kind, "fact_rows": _log_int(rng, 20_000, 4_000_000), "rows": rng.randint(20, 400),
                "strings": rng.random() < 0.5}
    if kind == "scan":
        strings = rng.random() < 0.5
        return {"kind": kind, "rows": _log_int(rng, 2_000, 1_000_000 if strings else 16_000_000),
                "sel": round(rng.uniform(0.01, 0.5), 3), "strings": strings, "filters": rng.randint(1, 2)}
    if kind == "lookup":
        return {"kind": kind, "build_rows": _log_int(rng, 1_000, 2_000_000),
                "probe_rows": _log_int(rng, 10_000, 10_000_000), "match": round(rng.uniform(0.1, 1.0), 3),
                "nulls": rng.random() < 0.5, "kept": rng.random() < 0.5}
    plain, dup = rng.random() < 0.25, rng.choice((1, 1, 3))
    lo = _log_int(rng, 1_000, 100_000)
    hi = _log_int(rng, lo, 200_000 if dup > 1 else 1_000_000 if plain else 4_000_000)
    return {"kind": kind, "n": _log_int(rng, 1, 6 if plain else 16 if dup > 1 else 64), "lo": lo, "hi": hi, "dup": dup,
            "plain": plain}


# ------------------------------------------------------------------ inputs --

class Gen:
    """Seeded columns, made on the GPU."""

    def __init__(self, seed: int):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(seed * 7919 + 17)

    def ints(self, n: int, lo: int, hi: int):
        return torch.randint(lo, hi, (n,), generator=self.g, device="cuda", dtype=torch.int64).int()

    def perm(self, n: int):
        return torch.randperm(n, generator=self.g, device="cuda").int()

    def valid(self, n: int, p_null: float):
        return torch.rand(n, generator=self.g, device="cuda") >= p_null

    def ranks(self, n: int, k: int, s: float):
        """n draws of a rank in [0, k), P(r) ~ (r + 1)^-s (s = 0: uniform)."""
        if s == 0:
            return torch.randint(0, k, (n,), generator=self.g, device="cuda", dtype=torch.int64)
        cdf = torch.arange(1, k + 1, device="cuda", dtype=torch.float64).pow_(-s).cumsum_(0)
        u = torch.rand(n, generator=self.g, device="cuda", dtype=torch.float64) * cdf[-1]
        return torch.searchsorted(cdf, u).clamp_(max=k - 1)

    def strings(self, n: int, lo: int, hi: int):
        """A VARCHAR column of printable strings of lo..hi bytes."""
        lens = torch.randint(lo, hi + 1, (n,), generator=self.g, device="cuda", dtype=torch.int64)
        offs = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
        torch.cumsum(lens, 0, out=offs[1:])
        data = torch.randint(0x20, 0x7F, (max(1, int(offs[-1])),), generator=self.g, device="cuda", dtype=torch.uint8)
        return hj.Column.varchar(data.cpu().numpy(), offs.cpu().numpy().astype(np.uint64))


def column(values, valid=None):
    """An INT32 column's host pages from device values."""
    return hj.Column.int32(values.cpu().numpy(), None if valid is None else valid.cpu().numpy().astype(np.uint8))


class State:
    """What a program keeps between calls; gives the engine's tables back when dropped."""

    def __init__(self, kind: str):
        self.kind, self.resident, self.table = kind, [], None

    def plan(self, plan, prepared: bool, max_rows: int, max_str: int = 64):
        """The plan over tables resident in HBM, its descriptor built once, and the result's
        buffers: max_rows rows, strings of max_str bytes at most."""
        for t in plan.inputs:
            r = engine().upload(t)
            if prepared:
                engine().prepare(r)
            self.resident.append(r)
        self.frozen = hj.Plan(plan.nodes, list(self.resident), plan.root).frozen()
        self.out = []
        for _, t in plan.nodes[plan.root][2]:
            pages = max_rows // 1984 + 1 if t == I else max_rows * (max_str + 3) // 7000 + max_rows // 4096 + 2
            self.out.append(torch.zeros((pages, hj.PAGE_SIZE), dtype=torch.uint8).pin_memory())
        return self

    def __del__(self):
        try:
            if self.table is not None:
                hj.lib().hj_table_free(self.table)
            for t in self.resident:
                engine().release(t)
        except Exception:  # at interpreter exit
            pass


def _chain(c: dict, g: Gen) -> State:
    sizes = [max(2, c["dim_rows"] >> (2 * i)) for i in range(c["rels"] - 1)]
    p = hj.Plan()

    def table(n, keys, fk_of):
        cols = [column(keys)] if keys is not None else []
        if fk_of:
            cols.append(column(g.ints(n, 0, fk_of)))
        cols.append(column(g.ints(n, 0, 2**31 - 1), g.valid(n, 0.05)))
        types = [I] * len(cols)
        if c["strings"]:
            cols.append(g.strings(n, 4, 40))
            types.append(V)
        p.new_input(hj.Table(n, cols))
        return p.new_scan_node(len(p.inputs) - 1, list(enumerate(types))), types

    cur, layout = table(c["rows"], None, sizes[0])       # fk, payload[, string]
    fk, keep = 0, list(range(1, len(layout)))            # positions: next foreign key, payloads kept
    for i, n in enumerate(sizes):
        last = i + 1 == len(sizes)
        scan, types = table(n, g.perm(n), 0 if last else sizes[i + 1])  # pk[, fk], payload[, string]
        base = len(layout)
        both = layout + types
        new_pay = [base + j for j in range(1 if last else 2, len(types))]
        out = ([] if last else [base + 1]) + keep + new_pay
        cur = p.new_join_node(False, cur, scan, fk, 0, [(j, both[j]) for j in out])
        layout, fk = [both[j] for j in out], 0
        keep = list(range(0 if last else 1, len(out)))
    p.root = cur
    return State("execute").plan(p, c["prepared"], c["rows"], 40)


def _funnel(c: dict, g: Gen) -> State:
    nf, nd, dup = c["fact_rows"], c["dim_rows"], c["dup"]
    dom = max(1, nd // dup)
    keys = g.perm(nd) if dup == 1 else g.ints(nd, 0, dom)
    spread = g.perm(dom).long()  # rank -> key, so that popular keys lie anywhere
    fk = spread[g.ranks(nf, dom, c["skew"])].int()
    ids = g.perm(nf)
    ns = min(c["sel_rows"], nf)
    p = hj.Plan()
    p.new_input(hj.Table(nd, [column(keys), column(g.ints(nd, 0, 2**31 - 1), g.valid(nd, 0.2))]))
    p.new_input(hj.Table(nf, [column(ids), column(fk), column(g.ints(nf, 0, 2**31 - 1), g.valid(nf, 0.2))]))
    p.new_input(hj.Table(ns, [column(ids[g.perm(nf)[:ns].long()]), column(g.ints(ns, 0, 100))]))
    dim = p.new_scan_node(0, [(0, I), (1, I)])
    fact = p.new_scan_node(1, [(0, I), (1, I), (2, I)])
    sel = p.new_scan_node(2, [(0, I), (1, I)])
    # dim.key, dim.pay, fact.id, fact.fk, fact.pay; a duplicate key's payloads differ, so only a
    # unique dimension shows them
    mid = p.new_join_node(True, dim, fact, 0, 1, [(2, I), (4, I), (1 if dup == 1 else 0, I)])
    p.root = p.new_join_node(True, mid, sel, 0, 0, [(0, I), (1, I), (2, I), (4, I)])
    return State("execute").plan(p, c["prepared"], ns if dup == 1 else 8 * dup * ns + 64)


def _fanout_rows(c: dict) -> float:
    """Result rows to expect: the fact rows of the popular keys."""
    nf, dom = c["fact_rows"], max(c["rows"] + RANK0, c["fact_rows"] // 4)
    w = np.arange(1, dom + 1, dtype=np.float64) ** -1.1
    return float(nf * w[RANK0:RANK0 + c["rows"]].sum() / w.sum())


def _fanout(c: dict, g: Gen) -> State:
    nf, n = c["fact_rows"], c["rows"]
    dom = max(n + RANK0, nf // 4)
    spread = g.perm(dom).long()
    p = hj.Plan()
    p.new_input(hj.Table(nf, [column(spread[g.ranks(nf, dom, 1.1)].int()), column(g.ints(nf, 0, 1000))]))
    cols = [column(spread[RANK0:RANK0 + n][g.perm(n).long()].int())]  # in any order
    cols.append(column(g.ints(n, 0, 2**31 - 1), g.valid(n, 0.2)))
    types = [I, I]
    if c["strings"]:
        cols.append(g.strings(n, 8, 64))
        types.append(V)
    p.new_input(hj.Table(n, cols))
    fact = p.new_scan_node(0, [(0, I)])
    short = p.new_scan_node(1, list(enumerate(types)))
    p.root = p.new_join_node(True, fact, short, 0, 0, [(1 + j, t) for j, t in enumerate(types)])
    return State("execute").plan(p, False, int(1.3 * _fanout_rows(c)) + 500)


def _scan(c: dict, g: Gen) -> State:
    n = c["rows"]
    cols = [column(g.ints(n, 0, 1000)), column(g.ints(n, 0, 2**31 - 1)),
            column(g.ints(n, 0, 2**31 - 1), g.valid(n, 0.2))]
    out = [(1, I), (2, I)]
    if c["strings"]:
        cols.append(g.strings(n, 8, 64))
        out.append((3, V))
    filters = [(0, hj.CMP_LT, int(round(1000 * c["sel"])))]
    if c["filters"] > 1:
        filters.append((2, hj.CMP_IS_NOT_NULL, 0))
    p = hj.Plan()
    p.new_input(hj.Table(n, cols))
    p.root = p.new_scan_node(0, out, filters)
    return State("execute").plan(p, False, min(n, int(1.2 * n * c["sel"]) + 200))


def _lookup(c: dict, g: Gen) -> State:
    nb, n = c["build_rows"], c["probe_rows"]
    s = State("lookup")
    s.keys = g.perm(nb)
    hit = torch.rand(n, generator=g.g, device="cuda") < c["match"]
    s.probe = g.ints(n, 0, nb) + torch.where(hit, 0, nb).int()
    s.valid = None
    if c["nulls"]:
        s.valid = torch.randint(-2**31, 2**31, ((n + 31) // 32,), generator=g.g, device="cuda", dtype=torch.int64)
        s.valid = (s.valid | torch.randint(-2**31, 2**31, s.valid.shape, generator=g.g, device="cuda")).int()
    s.stream = torch.cuda.ExternalStream(engine().stream)
    torch.cuda.synchronize()
    if c["kept"]:
        s.table = _build(s.keys)
    return s


def _build(keys):
    t = C.c_void_p()
    rc = hj.lib().hj_table_build(engine().handle, keys.data_ptr(), None, keys.numel(), -1, C.byref(t))
    assert rc == hj.HJ_OK, rc
    return t


def _batch(c: dict, g: Gen, seed: int) -> State:
    s = State("batch")
    s.mode = hj.BATCH_PLAIN if c["plain"] else hj.BATCH_PERSISTENT
    w = workloads.c4(n=c["n"], seed=seed % (1 << 31), lo=c["lo"], hi=c["hi"])
    s.wave = batch.generate(engine(), w, list(range(c["n"])), torch)
    if c["dup"] > 1:  # build keys repeat: about `dup` rows a key
        for inst in s.wave.instances:
            nb = inst[1][2]
            for ptr, _, n in inst:
                at = (ptr - s.wave.keep[0].data_ptr()) // 4
                s.wave.keep[0][at:at + n] = g.ints(n, 0, max(1, nb // c["dup"]))
        torch.cuda.synchronize()
    return s


def prepare(case: dict, seed: int) -> State:
    g = Gen(seed)
    if case["kind"] == "batch":
        return _batch(case, g, seed)
    return {"chain": _chain, "funnel": _funnel, "fanout": _fanout, "scan": _scan, "lookup": _lookup}[case["kind"]](case, g)


# -------------------------------------------------------------------- pass --

def run(s: State):
    e = engine()
    if s.kind == "execute":
        lib, rows, pages = hj.lib(), C.c_uint64(), C.c_uint64()
        r = e.execute_raw(s.frozen)
        lib.hj_result_shape(r, C.byref(rows), None)
        for i, buf in enumerate(s.out):
            lib.hj_result_column(r, i, None, C.byref(pages))
            assert pages.value <= buf.shape[0], (pages.value, buf.shape)
            rc = lib.hj_result_copy_contiguous(e.handle, r, i, buf.data_ptr())
            assert rc == hj.HJ_OK, rc
        e.free_result(r)
        return {"rows": rows.value, "columns": s.out}
    if s.kind == "batch":
        rows, sums, redo = e.batch_execute(s.wave.instances, s.mode)
        return {"rows": rows.view(np.int64), "sums": sums.view(np.int64), "recomputed": redo}
    n, found = s.probe.numel(), C.c_uint64()
    with torch.cuda.stream(s.stream):  # the program's own work in the engine's order
        table = s.table if s.table is not None else _build(s.keys)
        prow = torch.empty(n, dtype=torch.int32, device="cuda")
        brow = torch.empty(n, dtype=torch.int32, device="cuda")
        rc = hj.lib().hj_table_probe(e.handle, table, s.probe.data_ptr(),
                                     None if s.valid is None else s.valid.data_ptr(), n, prow.data_ptr(),
                                     brow.data_ptr(), n, C.byref(found))
        assert rc == hj.HJ_OK, rc
        if s.table is None:
            hj.lib().hj_table_free(table)
        m = found.value
        out = torch.full((n,), -1, dtype=torch.int32, device="cuda")
        out[prow[:m].long()] = brow[:m]
    return out


def exact(case: dict, seed: int):
    """Outputs are whole numbers and bytes, which stay equal: no value in 64 bits."""
    return None


def work(case: dict) -> dict:
    """Bytes of the inputs read once and of the result written once."""
    k = case["kind"]
    if k == "chain":
        s = 24 if case["strings"] else 0
        dims = sum(max(2, case["dim_rows"] >> (2 * i)) for i in range(case["rels"] - 1))
        b = dims * (12 + s) + case["rows"] * (8 + s) + case["rows"] * case["rels"] * (4 + s)
    elif k == "funnel":
        b = case["dim_rows"] * 8 + case["fact_rows"] * 12 + case["sel_rows"] * (8 + 16 * case["dup"])
    elif k == "fanout":
        s = 38 if case["strings"] else 0
        out = _fanout_rows(case)
        b = case["fact_rows"] * 4 + case["rows"] * (8 + s) + out * (8 + s)
    elif k == "scan":
        s = 38 if case["strings"] else 0
        kept = case["rows"] * case["sel"] * (0.8 if case["filters"] > 1 else 1.0)
        read = 4 if case["filters"] == 1 else 8
        b = case["rows"] * read + kept * (8 + s) + kept * (8 + s)
    elif k == "lookup":
        b = (0 if case["kept"] else 4 * case["build_rows"]) + 8 * case["build_rows"] + 8 * case["probe_rows"]
    else:  # mean of a log-uniform build size; two build relations on average beside the probe's ten-fold
        lo, hi = case["lo"], case["hi"]
        mean = (hi - lo) / math.log(hi / lo) if hi > lo else lo
        b = case["n"] * mean * 12 * 8
    return {"bytes": float(b), "flops": 0.0}
