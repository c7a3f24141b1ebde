"""Device memory that calls take beyond their inputs and results, each call in a
process of its own, where the memory that is in use is known."""
from __future__ import annotations

import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]
HEAD = """
import ctypes as C, sys
sys.path.insert(0, {root!r})
import numpy as np, torch
from __graft_entry__ import load
hj = load()
E, L = hj.Engine(0), hj.lib()
def free(): return torch.cuda.mem_get_info()[0]
def ints(n, v): return torch.full((n,), v, dtype=torch.int32, device="cuda")
"""


def run(code: str):
    out = subprocess.run([sys.executable, "-c", HEAD.format(root=str(ROOT)) + code], capture_output=True, text=True,
                         timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr


def test_batch_instance_with_an_empty_relation():
    """Its other relations, however large, are neither partitioned nor built on."""
    run("""
n = 50_000_000
big, small, none = ints(n, 3), ints(100, 3), ints(1, 3)
def rel(t, rows=None): return (t.data_ptr(), t.data_ptr(), t.numel() if rows is None else rows)
inst = [[rel(small), rel(small)], [rel(small), rel(big), rel(none, 0)], [rel(none, 0), rel(big)], [rel(small), rel(none, 0)]]
torch.cuda.synchronize()
E.batch_execute([inst[0]])
before = free()
rows, sums, redo = E.batch_execute(inst)
assert list(rows) == [100 * 100, 0, 0, 0] and sums[1] == sums[2] == sums[3] == 0 and redo == 0
assert before - free() < 4 * n, before - free()
""")


def test_selective_join_keeps_streams_of_its_result():
    """Two joins over 40M probe rows, few of which match: the row ids of the first take
    no more than its result while the second runs, so both together take a probe's lists
    and output streams once."""
    run("""
n = 40_000_000
a = np.zeros(n, np.int32); a[:1000] = np.arange(1, 1001)
few = np.arange(1, 1001, dtype=np.int32)
p = hj.Plan()
for cols, rows in (([few], 1000), ([a, a], n)):
    p.new_input(E.upload(hj.Table(rows, [hj.Column.int32(c) for c in cols])))
I = hj.INT32
def join():  # (few x big): big's two columns and few's
    s, b = p.new_scan_node(0, [(0, I)]), p.new_scan_node(1, [(0, I), (1, I)])
    return p.new_join_node(True, s, b, 0, 0, [(1, I), (2, I), (0, I)])
p.root = p.new_join_node(True, join(), join(), 0, 0, [(0, I), (3, I)])
first = free()
r = E.execute_raw(p)
assert E.stats(r)[2] == 3000
# a probe's lists are 36 bytes a row, its streams here 2 x 4 bytes for n + 2^24 rows; the decoded
# columns are read in place
assert first - free() < 36 * n + 8 * (n + (1 << 24)) + (300 << 20), first - free()
""")


@pytest.mark.parametrize("call", ["table_probe", "execute", "plain"])
def test_probe_without_room_for_streams_ahead(call):
    """With device memory for a probe's lists and its result, but not for output streams of
    the probe side's length beside them, the result is the same."""
    run("call = " + repr(call) + """
n, nb = 1 << 25, 1000
build, probe = ints(nb, 0), ints(n, -5)
build.copy_(torch.arange(nb)); probe[:300] = torch.arange(300, dtype=torch.int32)
torch.cuda.synchronize()
lists = 9 * 4 * n
def fill(room):
    global hold
    torch.cuda.synchronize()
    hold = torch.empty(free() - room, dtype=torch.uint8, device="cuda")
if call == "table_probe":
    t, nm = C.c_void_p(), C.c_uint64()
    assert L.hj_table_build(E.handle, build.data_ptr(), None, nb, -1, C.byref(t)) == 0
    op, ob = ints(1000, -1), ints(1000, -1)
    fill(lists + (230 << 20))  # (an array takes up to 16 MB more than its size; streams would take 256 MB)
    assert L.hj_table_probe(E.handle, t, probe.data_ptr(), None, n, op.data_ptr(), ob.data_ptr(), 1000, C.byref(nm)) == 0
    torch.cuda.synchronize()
    assert nm.value == 300 and bool((op[:300] == ob[:300]).all()) and int(op[:300].sum()) == 300 * 299 // 2
elif call == "execute":
    p, I = hj.Plan(), hj.INT32
    for t in (build, probe):
        p.new_input(E.upload(hj.Table(t.numel(), [hj.Column.int32(t.cpu().numpy())])))
    p.root = p.new_join_node(True, p.new_scan_node(0, [(0, I)]), p.new_scan_node(1, [(0, I)]), 0, 0, [(0, I), (1, I)])
    fill(lists + (360 << 20))  # (streams would take 400 MB)
    r = E.execute(p)
    v, ok = hj.decode_int32(r.columns[0])
    assert r.num_rows == 300 and sorted(v.tolist()) == list(range(300))
else:
    inst = [[(probe.data_ptr(), probe.data_ptr(), n), (build.data_ptr(), build.data_ptr(), nb)]]
    want, sums, _ = E.batch_execute(inst)  # (persistent: takes little)
    fill(lists + (230 << 20))
    rows, s2, _ = E.batch_execute(inst, hj.BATCH_PLAIN)
    assert rows[0] == want[0] == 300 and sums[0] == s2[0]
""")


def test_batch_of_many_small_instances():
    """What an instance takes beside its rows does not grow past them: 200,000 instances of
    10 build rows, each with a key that repeats."""
    run("""
n = 200_000
k = torch.arange(10, dtype=torch.int32, device="cuda")
k[9] = 3
one = [(k.data_ptr(), k.data_ptr(), 10)] * 3
torch.cuda.synchronize()
E.batch_execute([one])
before = free()
rows, sums, redo = E.batch_execute([one] * n)
assert set(rows) == {8 + 2 * 2 * 2} and len(set(sums)) == 1 and redo == 0
assert before - free() < n * 1600, before - free()
""")
