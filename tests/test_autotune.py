"""Launch-shape autotuner (fz_autotune, fz_group_autotune, fz_set_kz_chunk): tuning mid-solve
leaves the solve exactly where it was, and the results do not depend on the tile depth. Every
comparison is bit for bit against an untuned run of the same steps, with a second source placed
inside the obstacle (a cell the stage kernels skip, whose stale output accumulates the source)."""
import numpy as np
import pytest

from tests.helpers import small_room

# the second source sits inside the obstacle of small_room ((9,7,5)-(14,12,9) in room cells)
SOURCES = np.array([[6, 6, 12], [14, 12, 10]], np.int32)


def _solver(cfg, precision="fp32", batch=1, steps=40):
    from fases_b200 import Solver, params
    s = Solver(params(h=cfg["h"], c=cfg["c"], rho=cfg["rho"], dt=cfg["dt"], pml=cfg["pml"],
                      pml_cells=cfg["pml_cells"], precision=precision, batch=batch))
    s.load_geometry(cfg["scene"].S, cfg["scene"].oid)
    m = cfg["materials"]
    s.set_materials(m["Rinf"], m["A"], m["zeta"], m["B"], m["Cc"], m["alpha"], m["beta"])
    s.set_sources(SOURCES, np.full(len(SOURCES), cfg["sval"][0]), cfg["src_opt"], u_s=cfg["u_s"])
    s.set_receivers(cfg["recs"], steps)
    if cfg["p0"] is not None:
        p0 = cfg["p0"] if batch == 1 else np.stack([cfg["p0"]] * batch)
        s.set_fields(p=p0)
    return s


def test_tuner_entry_points_check_arguments():
    from fases_b200 import _abi
    L = _abi.lib()
    assert L.fz_autotune(None, 3, None, None) == _abi.FZ_EINVAL
    assert L.fz_group_autotune(None, 3, None, None) == _abi.FZ_EINVAL
    assert L.fz_set_kz_chunk(None, 4) == _abi.FZ_EINVAL
    assert L.fz_set_z_schedule(None, None, 0) == _abi.FZ_EINVAL


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_tuning_mid_solve_changes_nothing(precision):
    cfg = small_room(seed=7, pml=(1, 0, 1, 0, 0, 1), steps=40)
    ref = _solver(cfg, precision)
    ref.run(40)
    ir_ref, f_ref = ref.ir(), ref.fields()
    ref.close()
    s = _solver(cfg, precision)
    s.run(13)
    depth, ms = s.autotune(reps=2)
    cur, heur = s.kz_chunk()
    assert depth == cur and depth >= 1 and heur >= 1 and ms > 0
    s.run(11)
    s.set_kz_chunk(5)  # an odd depth that leaves a short last chunk
    assert s.kz_chunk()[0] == 5
    s.run(7)
    nzi = s.shape[0] - 6
    sched = [nzi - 3, 2, 1] if nzi > 3 else [nzi]  # chunks of unequal length, longest first
    s.set_z_schedule(sched)
    assert s.z_schedule() == sched
    s.run(9)
    assert np.array_equal(s.ir(), ir_ref)
    for a, b in zip(s.fields(), f_ref):
        assert np.array_equal(a, b)
    s.close()


@pytest.mark.gpu
def test_tuning_batched_and_grouped_solves():
    from fases_b200 import Group
    cfg = small_room(seed=9, pml=(0, 0, 1, 0, 0, 0), steps=30)
    ref = _solver(cfg, batch=3, steps=30)
    ref.run(30)
    ir_ref = ref.ir()
    ref.close()
    b = _solver(cfg, batch=3, steps=30)
    b.run(10)
    b.autotune(reps=2)
    b.run(20)
    assert np.array_equal(b.ir(), ir_ref)
    b.close()
    rooms = [(26, 22, 18), (30, 20, 16), (20, 24, 22)]
    cfgs = [small_room(seed=30 + q, room=r, steps=30) for q, r in enumerate(rooms)]
    solos = []
    for c in cfgs:
        s = _solver(c, steps=30)
        s.run(30)
        solos.append(s.ir())
        s.close()
    members = [_solver(c, steps=30) for c in cfgs]
    with Group(members) as g:
        g.run(10)
        depth, ms = g.autotune(reps=2)
        assert depth >= 0 and ms > 0
        g.run(20)
        for s, r in zip(members, solos):
            assert np.array_equal(s.ir(), r)
    for s in members:
        s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("branches", [0, -1])
def test_untuned_group_chooses_for_all_rooms_together(branches):
    """Sixteen rooms of 48^3 fill the GPU together, so the launches that suit one of them alone (one-plane
    chunks, the direct kernel) are not theirs: an untuned group takes at most a quarter longer than one
    whose members are set to eight-plane chunks (with the rooms' own choices it took 1.5 and 2.2 times as
    long), and gives the same traces. Alone, a member runs as it would without the group."""
    from fases_b200 import Group
    cfgs = [small_room(seed=50 + q, room=(48, 48, 48), steps=200) for q in range(16)]

    def step_us(depth):
        members = [_solver(c, steps=cfgs[0]["steps"]) for c in cfgs]
        own = [s.z_schedule() for s in members]
        if depth:
            for s in members:
                s.set_kz_chunk(depth)
        with Group(members) as g:
            g.set_branches(branches)
            g.run(40)
            us = min(g.run_timed(40) for _ in range(4)) / 40 * 1e3
        ir = [s.ir() for s in members]
        if not depth:
            assert [s.z_schedule() for s in members] == own
        for s in members:
            s.close()
        return us, ir

    default, ir = step_us(0)
    deep, ir_deep = step_us(8)
    assert default <= 1.25 * deep, (default, deep)
    for a, b in zip(ir, ir_deep):
        assert np.array_equal(a, b)


def _band_launches(s):
    s.profile(True)
    s.run(2)
    n = s.profile_read()["band"][1]
    s.profile(False)
    return n


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_tuned_launches_come_back_from_the_depth_and_the_schedule(precision):
    """In a room this small the direct kernel (no band launches) wins by far; the depth that the tuner
    returns, and the schedule, select it again on another handle, and any other depth does not."""
    cfg = small_room(seed=7, steps=40)
    s = _solver(cfg, precision)
    for _ in range(5):  # (the host may be held up in the middle of a trial)
        depth, _ = s.autotune(reps=20)
        sched = s.z_schedule()
        bands = _band_launches(s)
        if bands == 0:
            break
    assert bands == 0
    other = 4 if depth != 4 else 5
    for select, launches in ((lambda x: x.set_kz_chunk(depth), 0), (lambda x: x.set_z_schedule(sched), 0),
                             (lambda x: x.set_kz_chunk(0), 0), (lambda x: x.set_kz_chunk(other), 6)):
        t = _solver(cfg, precision)
        t.set_kz_chunk(other)
        select(t)
        assert _band_launches(t) == launches
        t.close()
    s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("room", [(26, 22, 18), (71, 53, 47)])
def test_tuning_is_not_entered_into_a_profile(room):
    s = _solver(small_room(seed=7, room=room, steps=40))
    s.profile(True)
    s.run(1)
    s.profile_read()
    s.autotune(reps=2)
    assert all(n == 0 for _, n in s.profile_read().values())
    s.run(1)
    assert s.profile_read()["stage0"][1] == 1
    s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("room,precision,direct", [((256, 256), "fp32", True), ((500, 400), "fp32", False),
                                                   ((500, 400), "fp64", True), ((640, 500), "fp64", False)])
def test_planar_rooms_take_the_faster_kernel(room, precision, direct):
    """Either side of the line between the direct and the marching kernel, which lies lower in FP32 (500 x 400:
    34.5 us a step direct, 33.2 marching; FP64 39 and 47). The direct kernel launches no bands."""
    from fases_b200 import Solver, params, scenes
    from fases_b200 import materials as mats
    sc = scenes.box_room_2d(room, 0.05)
    s = Solver(params(h=0.05, precision=precision, two_d=True))
    s.load_geometry(sc.S, sc.oid)
    m = mats.pack([mats.rigid(0.9)] * 4)
    s.set_materials(m["Rinf"], m["A"], m["zeta"], m["B"], m["Cc"], m["alpha"], m["beta"])
    assert _band_launches(s) == (0 if direct else 6)
    s.close()
