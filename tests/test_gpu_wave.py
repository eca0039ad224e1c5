"""GPU test of the hyperplane-column sweep (csrc/sweep_wave.cu, the default schedule) against the
other schedules, bit for bit: boxes narrower than a column, boxes that end inside one and span
several, octants of 8, 64 and 216 velocities (216: a short last chunk of velocities). FP64 against the
per-node hyperplanes (which equal the oracle), FP32 against the tile diagonals, whose update
is the same operations (tolerance 0 in both)."""
import numpy as np
import pytest

import piks3d_b200 as pk
from conftest import base_params
from oracle import SlabOracle
from piks3d_b200 import images
from piks3d_b200.slab import LocalSlabs

pytestmark = pytest.mark.gpu

BOXES = [((4, 5, 6), 0.7), ((11, 10, 9), 0.5), ((12, 13, 40), 0.5), ((27, 8, 23), 0.4), ((21, 22, 5), 0.85)]


@pytest.mark.parametrize("prec", [pk.PREC_FP64, pk.PREC_FP32])
@pytest.mark.parametrize("nf", [2, 4, 6])
@pytest.mark.parametrize("box,porosity", BOXES)
def test_columns_equal_the_other_schedules(box, porosity, nf, prec):
    nx, ny, nz = box
    img = images.sphere_pack(max(box), porosity, 1.2, 3.0, seed=11)[:nz, :ny, :nx]
    p = base_params(max(box), Nx=nx, Ny=ny, Nz=nz, Nc_fundamental=nf, Kn=0.6, wallExtOrder=1, fluidlayer=1)
    out = []
    for wave in (True, False):
        with pk.Solver(p, device=0) as s:
            s.set_precision(prec)
            if wave:
                s.setup_physical_grid(img)
                assert s.schedule()["launch"] == pk.SCHED_WAVE
            else:
                s.set_tiles(*((0, 0, 0) if prec == pk.PREC_FP64 else (4, 4, 4)))
                s.setup_physical_grid(img)
            s.iterate(5)
            out.append((s.get_f()[0], s.chk_converge()))
    assert np.array_equal(out[0][0], out[1][0]) and out[0][1] == out[1][1]


def test_switching_schedules_keeps_the_iteration():
    """A context that moves between the columns and the tile schedules between iterations, and
    switches precision on the way, gives the values of one that does not."""
    img = images.sphere_pack(18, 0.5, 1.5, 3.5, seed=2)
    p = base_params(18, Nc_fundamental=4, Kn=0.5, wallExtOrder=1)
    out = []
    for moves in (True, False):
        with pk.Solver(p, device=0) as s:
            s.set_precision(pk.PREC_FP32)
            s.setup_physical_grid(img)
            for sched in (pk.SCHED_TILE_DATAFLOW, pk.SCHED_WAVE, pk.SCHED_TILE_COLUMNS, pk.SCHED_WAVE):
                if moves:
                    s.set_schedule(sched)
                s.iterate(4)
                if sched == pk.SCHED_TILE_COLUMNS:
                    s.set_precision(pk.PREC_FP64)
            out.append((s.get_f()[0], s.chk_converge()))
    assert np.array_equal(out[0][0], out[1][0]) and out[0][1] == out[1][1]


@pytest.mark.parametrize("own", [None, (4, 4, 4), (0, 0, 0)])
def test_autotune_without_a_usable_candidate_keeps_the_schedule(own):
    """16^3 tiles of this box need more rows than shared memory holds. An autotune call that is given
    nothing else reports that; the context then iterates on the schedule it had (columns, tiles or
    nodes), from the state of a set-up, as one that was never tuned."""
    img = images.sphere_pack(20, 0.45, 1.5, 3.0, seed=8)
    p = base_params(20, Nc_fundamental=4, Kn=0.5, wallExtOrder=1)
    out = []
    for tune in (True, False):
        with pk.Solver(p, device=0) as s:
            if own:
                s.set_tiles(*own)
            s.setup_physical_grid(img)
            before = s.schedule()
            if tune:
                with pytest.raises(pk.PiksError, match="candidate"):
                    s.autotune([(16, 16, 16, pk.SCHED_TILE_DIAGONALS), (16, 16, 16, pk.SCHED_TILE_DATAFLOW)], sweeps=1)
                assert s.schedule() == before
            s.iterate(4)
            out.append((s.get_f()[0], s.chk_converge()))
    assert np.array_equal(out[0][0], out[1][0]) and out[0][1] == out[1][1]


def test_tile_diagonals_by_name_move_to_the_fp64_shape():
    """Tile diagonals asked for by name, without a shape: FP32 tiles of 4x4x4 that move to 8x4x4 at
    the switch to FP64 and give the columns' values."""
    img = images.sphere_pack(16, 0.5, 1.5, 3.5, seed=1)
    p = base_params(16, Nc_fundamental=4, Kn=0.5, fluidlayer=2)
    out = []
    for sched in (pk.SCHED_TILE_DIAGONALS, pk.SCHED_WAVE):
        with pk.Solver(p, device=0) as s:
            s.set_schedule(sched)
            s.set_precision(pk.PREC_FP32)
            s.setup_physical_grid(img)
            assert s.schedule()["launch"] == sched and s.schedule()["TX"] == 4
            s.iterate(6)
            s.set_precision(pk.PREC_FP64)
            assert s.schedule()["launch"] == sched and s.schedule()["TX"] == 8
            s.iterate(5)
            out.append((s.get_f()[0], s.chk_converge()))
    assert np.array_equal(out[0][0], out[1][0]) and out[0][1] == out[1][1]


@pytest.mark.parametrize("sched", [pk.SCHED_TILE_DIAGONALS, pk.SCHED_WAVE])
@pytest.mark.parametrize("n", [2, 3])
def test_slabs_by_schedule_equal_the_slab_oracle(n, sched):
    img = images.sphere_pack(16, 0.45, 1.2, 3.0, seed=2)
    p = base_params(16, wallExtOrder=1, Nc_fundamental=4)
    ls = LocalSlabs(p, img, n, schedule=sched)
    so = SlabOracle(p, img.tobytes(), n, nthreads=8)
    assert all(s.schedule()["launch"] == sched and s.schedule()["tiles"] for s in ls.solvers)
    for _ in range(3):
        ls.iterate(1)
        so.iterate(1)
    for a, b in zip(so.macro(), ls.macro()):
        assert np.array_equal(a, b)
    assert ls.chk_converge() == so.chk_converge()
    ls.close()
    so.close()


@pytest.mark.parametrize("nf,prec", [(4, pk.PREC_FP64), (4, pk.PREC_FP32), (2, pk.PREC_FP32)])
def test_column_waits_give_up_and_the_context_stays_usable(nf, prec):
    """A column that waits for a hyperplane nobody publishes (no fault, trap or hang): its wait runs
    out, alone and in a batch, the sweep ends with the error reported, and the context, set up
    again, iterates as a fresh one. 512 velocities: two chunks an octant in FP64, so that the
    consumers change their class table on the way."""
    img = images.sphere_pack(33, 0.6, 1.5, 3.5, seed=9)
    p = base_params(33, Nc_fundamental=nf, Kn=0.8, wallExtOrder=1)
    with pk.Solver(p, device=0) as s:
        s.set_precision(prec)
        s.setup_physical_grid(img)
        assert s.schedule()["launch"] == pk.SCHED_WAVE and s.schedule()["columns"] > 8
        s.iterate(3)
        sec = s.selftest_wait_timeout()
        print("column sweep with a wait that nothing ends: %.3f s" % sec)
        assert 0.5 < sec < 10.0
        s.synchronize()
        s.setup_physical_grid(img)
        s.iterate(5)
        a = (s.get_f()[0], s.chk_converge())
    with pk.Solver(p, device=0) as r:
        r.set_precision(prec)
        r.setup_physical_grid(img)
        r.iterate(5)
        b = (r.get_f()[0], r.chk_converge())
    assert np.array_equal(a[0], b[0]) and a[1] == b[1]


def test_wait_selftest_refuses_a_box_of_one_column():
    img = images.sphere_pack(8, 0.6, 1.2, 2.5, seed=9)
    with pk.Solver(base_params(8, Nc_fundamental=4), device=0) as s:
        s.setup_physical_grid(img)
        with pytest.raises(pk.PiksError, match="waits for another"):
            s.selftest_wait_timeout()


def _diagonal_plates(n):
    """Solid and fluid plates of five cells each across one octant's direction: a whole hyperplane of
    a column becomes fluid at once behind a solid one, and its tasks read most rows (the ring holds
    685 rows beside the longer lists, 686 in every ordinary image, and a window of three batches 680)."""
    i = np.indices((n, n, n))
    return (((i.sum(0) + 3) % 10) < 5).astype(np.uint8)


def _run(img, prec, steps, nodes=False, **kw):
    with pk.Solver(base_params(img.shape[0], Kn=0.6, wallExtOrder=1, **kw), device=0) as s:
        s.set_precision(prec)
        if nodes:
            s.set_tiles(*((0, 0, 0) if prec == pk.PREC_FP64 else (4, 4, 4)))
        s.setup_physical_grid(img)
        assert (s.schedule()["launch"] == pk.SCHED_WAVE) == (not nodes)
        s.iterate(steps)
        return s.get_f()[0], s.chk_converge(), s.schedule()["ring"]


@pytest.mark.parametrize("prec", [pk.PREC_FP64, pk.PREC_FP32])
def test_batch_of_members_with_different_rings(prec):
    """Members whose rings differ: in FP32 one launch holds both and changes the ring between items,
    in FP64 they go to launches of their own. Every member equals its run alone, which equals the
    other schedule's."""
    imgs = [images.sphere_pack(24, 0.5, 1.5, 3.5, seed=7), _diagonal_plates(24), images.sphere_pack(21, 0.6, 1.5, 3.0, seed=8)]
    alone = [_run(i, prec, 4, Nc_fundamental=4) for i in imgs]
    assert len({a[2] for a in alone}) == 2
    other = _run(imgs[1], prec, 4, nodes=True, Nc_fundamental=4)
    assert np.array_equal(alone[1][0], other[0]) and alone[1][1] == other[1]
    members = []
    with pk.Batch(device=0) as b:
        for img in imgs:
            s = pk.Solver(base_params(img.shape[0], Kn=0.6, wallExtOrder=1, Nc_fundamental=4), device=0)
            s.set_precision(prec)
            s.setup_physical_grid(img)
            members.append(s)
            b.add(s)
        b.iterate(4)
        mass, perm, err = b.chk_converge()
    for k, s in enumerate(members):
        assert np.array_equal(s.get_f()[0], alone[k][0]) and (mass[k], perm[k], err[k]) == alone[k][1]
        s.close()


@pytest.mark.parametrize("prec", [pk.PREC_FP64, pk.PREC_FP32])
@pytest.mark.parametrize("nf", [8, 12, 16])
def test_columns_of_many_velocity_chunks(nf, prec):
    """Octants of 512, 1728 and 4096 velocities, up to 128 chunks a column, in a box of several columns."""
    img = images.sphere_pack(14, 0.6, 1.2, 2.5, seed=21)[:7, :14, :14]
    out = []
    for wave in (True, False):
        with pk.Solver(base_params(14, Nz=7, Nc_fundamental=nf, Kn=2.0, wallExtOrder=1), device=0) as s:
            s.set_precision(prec)
            if not wave:
                s.set_tiles(*((0, 0, 0) if prec == pk.PREC_FP64 else (4, 4, 4)))
            s.setup_physical_grid(img)
            s.iterate(2)
            out.append((s.get_f()[0], s.chk_converge(), s.schedule()["columns"]))
    assert out[0][2] > 8 and out[1][2] == 0
    assert np.array_equal(out[0][0], out[1][0]) and out[0][1] == out[1][1]


@pytest.mark.parametrize("prec", [pk.PREC_FP64, pk.PREC_FP32])
def test_column_graph_replay_equals_plain_launches(prec):
    """Per-kernel timing launches plainly; otherwise iterations from the third on replay graphs."""
    img = images.sphere_pack(22, 0.5, 1.5, 3.5, seed=12)
    out = []
    for plain in (True, False):
        with pk.Solver(base_params(22, Nc_fundamental=4, Kn=0.5, wallExtOrder=1), device=0) as s:
            s.set_precision(prec)
            s.setup_physical_grid(img)
            s.enable_timing(plain)
            s.iterate(9)
            out.append((s.get_f()[0], s.chk_converge()))
    assert np.array_equal(out[0][0], out[1][0]) and out[0][1] == out[1][1]
