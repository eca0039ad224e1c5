"""CPU test of the hyperplane-column sweep schedule (csrc/wave.cpp): the schedule is replayed in
numpy as the kernel runs it - rows copied into a ring of exactly its size as soon as the ring's
rule allows (overwriting what it overwrites), tasks reading ring slots only, columns one after
another in their listed order - and every swept row must equal the per-node task list's result
bit for bit."""
import os
import re
import subprocess
import sys

import numpy as np
import pytest

import piks3d_b200 as pk
from conftest import base_params
from piks3d_b200 import images

FW = 1 << 30


def _update(own, reads, flags):
    """A stand-in for the update that depends on every operand and its place."""
    c = (0.31, -0.07, 0.23, -0.05, 0.19, -0.03)
    out = 0.4 * own + 0.01
    for k, r in enumerate(reads):
        out = out + c[k] * r
    return out * (1.0 + 0.125 * (flags & 1) + 0.25 * (flags >> 1 & 1) + 0.375 * (flags >> 2 & 1))


def _replay(s, f):
    A, B, R, task_ring, win, max_rows = s.geometry_array("wave_info").tolist()
    rows, tasks = s.geometry_array("wave_rows"), s.geometry_array("wave_tasks").reshape(-1, 4)
    batch, cols = s.geometry_array("wave_batch").reshape(-1, 4), s.geometry_array("wave_cols").reshape(-1, 8)
    order = s.geometry_array("wave_col_list")
    assert win <= R and sorted(order.tolist()) == list(range(len(cols)))
    finished = set()
    for col in order.tolist():
        b0, nb, octant, s0, upx, upy = cols[col, :6].tolist()
        for up in (upx, upy):
            assert up < 0 or up in finished      # every upwind column comes first
        ring = np.full(R + 1, np.nan)
        ring[0] = 0.0
        assert nb % 4 == 0                       # batches are requested in groups of four
        for g in range(b0, b0 + nb, 4):
            assert sum(-(-(int(b[2]) & 0xFFFF) // 4) * 4 for b in batch[g:g + 4]) <= max_rows
            assert all(batch[g + i + 1, 0] == batch[g + i, 0] + -(-(int(batch[g + i, 2]) & 0xFFFF) // 4) and
                       batch[g + i + 1, 1] == batch[g + i, 1] + (int(batch[g + i, 2]) >> 16) for i in range(3))
        sizes = [int(b[2]) & 0xFFFF for b in batch[b0:b0 + nb]]
        slots0 = [(int(b[3]) >> 16) & 0xFFFF for b in batch[b0:b0 + nb]]
        start, pos = [], 0                       # ring positions without wrapping
        for n, slot0 in zip(sizes, slots0):
            assert slot0 == 1 + pos % R
            start.append(pos)
            pos += n
        staged = 0
        for k in range(nb):
            # stage every batch the rule allows: batch j may go in once it overwrites nothing
            # that batches from k - 2 on (none after k - 1 is complete) read
            while staged < nb and start[staged] + sizes[staged] - start[max(0, k - 2)] <= R:
                x, t0, z, w = (int(v) for v in batch[b0 + staged])
                n, nt = z & 0xFFFF, (z >> 16) & 0xFFFF
                assert 4 * nt <= task_ring
                ring[1 + (start[staged] + np.arange(n)) % R] = f[rows[4 * x:4 * x + n]]
                staged += 1
            assert staged > k                    # three batches always fit
            x, t0, z, w = (int(v) for v in batch[b0 + k])
            nt, slot0 = (z >> 16) & 0xFFFF, (w >> 16) & 0xFFFF
            new = []
            for t in range(nt):
                rec = tasks[t0 + t].astype(np.int64) & 0xFFFFFFFF
                node, fl = int(rec[0]) & ((1 << 27) - 1), int(rec[0]) >> 27
                assert int(rows[4 * x + t]) == node * 8 + octant
                slots = [int(v) for q in rec[1:] for v in (q & 0xFFFF, q >> 16)]
                slot = slot0 + t - (R if slot0 + t > R else 0)
                new.append((slot, node * 8 + octant, _update(ring[slot], ring[slots], fl)))
            for slot, row, v in new:
                ring[slot] = v
                f[row] = v
        finished.add(col)
    return f


@pytest.mark.parametrize("n,kw", [((14, 14, 14), {}), ((21, 9, 17), dict(fluidlayer=2)), ((9, 30, 8), dict(Nc_fundamental=4)),
                                  ((33, 19, 12), dict(block_repy=2))])
def test_columns_replay_the_per_node_tasks(n, kw):
    nx, ny, nz = n
    m = max(n)
    img = np.ascontiguousarray(images.sphere_pack(m, 0.5, 1.2, 3.5, seed=17)[:nz, :ny, :nx])
    s = pk.Solver(base_params(m, Nx=nx, Ny=ny, Nz=nz, **kw), device=-1)
    s.setup_physical_grid(img)
    nn, nc = s.info()["nNodes"], s.info()["nCorner"]
    half = 8 * nn                                # the corner rows follow the nodes' rows
    start = np.random.default_rng(3).standard_normal(half + 8 * nc)
    want = start.copy()
    for t in s.geometry_array("tasks").reshape(-1, 8).tolist():
        reads = [0.0 if c < 0 else want[(c & ~FW) + (half if c & FW else 0)] for c in t[2:]]
        row = t[0] * 8 + (t[1] & 7)
        want[row] = _update(want[row], reads, t[1] >> 3)
    got = _replay(s, start.copy())
    assert np.array_equal(got, want)
    s.close()


def test_columns_replay_a_nearly_full_ring():
    """Plates across an octant's direction: a hyperplane of a column is fluid as a whole behind a
    solid one, a window of three batches takes 680 of the ring's 685 rows, and the lists are longer
    than the rows every context reserves for them (which costs the ring its 686th)."""
    n = 24
    img = (((np.indices((n, n, n)).sum(0) + 3) % 10) < 5).astype(np.uint8)
    s = pk.Solver(base_params(n, Nc_fundamental=4, wallExtOrder=1), device=-1)
    s.setup_physical_grid(img)
    assert s.geometry_array("wave_info").tolist() == [10, 10, 685, 1200, 680, 816]
    half = 8 * s.info()["nNodes"]
    start = np.random.default_rng(3).standard_normal(half + 8 * s.info()["nCorner"])
    want = start.copy()
    for t in s.geometry_array("tasks").reshape(-1, 8).tolist():
        reads = [0.0 if c < 0 else want[(c & ~FW) + (half if c & FW else 0)] for c in t[2:]]
        row = t[0] * 8 + (t[1] & 7)
        want[row] = _update(want[row], reads, t[1] >> 3)
    assert np.array_equal(_replay(s, start.copy()), want)
    s.close()


def test_warps_that_may_leave_meet_on_mbarriers_only():
    """Warps of the column kernel leave one by one once a bounded wait has given up. A counted
    barrier after that point would wait for the ones that left, without a limit: the kernel's only
    one is the __syncthreads() before its warps take up their roles."""
    src = open(os.path.join(os.path.dirname(pk.__file__), "csrc", "sweep_wave.cu")).read()
    code = re.sub(r"//[^\n]*", "", src)
    counted = re.findall(r"__syncthreads|\bbar\.(?:sync|red|arrive)|\bbarrier\.(?:cta\.)?(?:sync|red|arrive)|__barrier_sync", code)
    assert counted == ["__syncthreads"]
    kernel = code[code.index("k_wave_sweep(const DevState a"):]
    assert kernel.index("__syncthreads") < kernel.index("setmaxnreg")


def test_schedule_reports_what_is_in_use():
    """The getter describes the schedule that the context iterates and builds nothing: no tile jobs
    on a context that marches columns, and no column schedule named where another one runs."""
    img = images.sphere_pack(24, 0.5, 1.5, 3.5, seed=4)
    s = pk.Solver(base_params(24), device=-1)
    s.setup_physical_grid(img)
    sch = s.schedule()
    A, B, ring = s.geometry_array("wave_info").tolist()[:3]
    assert sch["launch"] == pk.SCHED_WAVE and sch["tiles"] and sch["jobs"] == 0 and sch["max_slots"] == 0
    assert (sch["cross_section"], sch["ring"], sch["columns"]) == ((A, B), ring, len(s.geometry_array("wave_cols")) // 8)
    s.set_tiles(4, 4, 4)                         # from the next set-up on
    assert s.schedule()["launch"] == pk.SCHED_WAVE and s.schedule()["columns"] == sch["columns"]
    s.setup_physical_grid(img)
    sch = s.schedule()
    assert sch["launch"] == pk.SCHED_TILE_DIAGONALS and sch["jobs"] > 0 and (sch["cross_section"], sch["columns"]) == ((0, 0), 0)
    s.close()
    s = pk.Solver(base_params(12), device=-1)
    s.setup_physical_grid(np.ones((12, 12, 12), np.uint8))   # nothing to sweep: no columns are built
    assert s.schedule()["launch"] != pk.SCHED_WAVE and s.schedule()["columns"] == 0
    s.close()


_NO_THREADS = """
import hashlib, os, resource, sys
sys.path[:0] = [%r, %r]
import numpy as np
import piks3d_b200 as pk
from conftest import base_params
from piks3d_b200 import images
img = images.sphere_pack(30, 0.5, 1.5, 3.5, seed=4)
def digests():
    out = []
    for tiles in (None, (4, 4, 4)):
        s = pk.Solver(base_params(30, Nc_fundamental=4), device=-1)
        if tiles:
            s.set_tiles(*tiles)
        s.setup_physical_grid(img)
        for name in ("tasks", "tile_rows", "tile_tasks") + (() if tiles else ("wave_rows", "wave_tasks", "wave_batch", "wave_cols")):
            out.append(hashlib.sha256(s.geometry_array(name).tobytes()).hexdigest())
        s.close()
    return out
want = digests()
if os.getuid() == 0:
    os.setuid(65534)                   # the limit does not hold for root
resource.setrlimit(resource.RLIMIT_NPROC, (0, 0))
import threading
try:
    threading.Thread(target=int).start()
    print("unlimited")
except RuntimeError:
    print("limited")
print("same" if digests() == want else "different")
"""


def test_setup_without_threads_to_be_had():
    """A process that may start no thread sets images up on the one it has, with the same result."""
    here = os.path.dirname(os.path.abspath(__file__))
    r = subprocess.run([sys.executable, "-c", _NO_THREADS % (os.path.dirname(here), here)], capture_output=True, text=True,
                       timeout=300)
    out = r.stdout.split()
    if out[:1] == ["unlimited"]:
        pytest.skip("the thread limit does not hold here")
    assert r.returncode == 0 and out == ["limited", "same"], (r.returncode, r.stdout, r.stderr[-800:])
