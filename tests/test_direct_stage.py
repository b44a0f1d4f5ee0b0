"""The direct stage kernel of small rooms (fz_direct.cu) against the marching kernel: the same
arithmetic per cell, so traces and fields agree bit for bit. Shapes at the edges of its tiles (30
cells of a row per warp, 4 rows per CTA, planar marches of one row and of two), every pole form of the band,
cPML on any face, sources in air and in skipped cells, batches and planar rooms."""
import numpy as np
import pytest

from fases_b200 import Solver, params
from fases_b200 import materials as mats
from fases_b200 import scenes


def _solve(room, precision, depth, K=2, L=2, pml=(0, 0, 1, 0, 0, 0), batch=1, two_d=False, steps=13):
    h, c, rho = 0.05, 343.0, 1.2
    rng = np.random.default_rng(5)
    dt = 0.5 * h / c
    sc = scenes.box_room_2d(room[:2], h) if two_d else scenes.box_room(room, h)
    walls = [mats.random_passive(rng, dt, c / (4 * h), K=K, L=L) for _ in range(4 if two_d else 6)]
    m = mats.pack(walls, K=max(K, 1), L=max(L, 1))
    s = Solver(params(h=h, c=c, rho=rho, dt=dt, pml=pml, pml_cells=4, precision=precision, two_d=two_d, batch=batch))
    s.load_geometry(sc.S, sc.oid)
    s.set_materials(m["Rinf"], m["A"], m["zeta"], m["B"], m["Cc"], m["alpha"], m["beta"])
    k = 3 if two_d else 3 + room[2] // 2
    air, skipped = [3 + room[0] // 2, 3 + room[1] // 2, k], [3, 3, k]  # S < h at the corner cell
    s.set_sources(np.array([air, skipped], np.int32), np.array([1e-3, 2e-3]), 0,
                  u_s=np.sin(0.2 * np.arange(2 * steps + 3)))
    if batch > 1:
        s.set_source_members(np.array([batch - 1, 0], np.int32))
    s.set_receivers(np.array([[4, 4, k], [2 + room[0], 2 + room[1], k]], np.int32), steps)
    if batch == 1:
        p0 = np.zeros(sc.shape)
        g = (slice(3, 4) if two_d else slice(3, -3), slice(3, -3), slice(3, -3))
        p0[g] = rng.standard_normal(p0[g].shape)
        s.set_fields(p=p0)
    if depth:
        s.set_kz_chunk(depth)  # an explicit depth selects the marching kernel
    s.run(steps)
    out = [s.ir(), s.vel()] + list(s.fields())
    s.close()
    return out


CASES = [
    ((16, 9, 8), {}), ((29, 8, 7), {}), ((30, 11, 9), {}), ((31, 10, 9), {"pml": (1, 1, 1, 1, 1, 1)}),
    ((61, 33, 20), {}), ((26, 22, 18), {"K": 4, "L": 3}), ((26, 22, 18), {"K": 6, "L": 1, "pml": (0, 1, 0, 0, 1, 0)}),
    ((26, 22, 18), {"K": 0, "L": 0}), ((20, 15, 11), {"batch": 3}), ((90, 1, 40), {}), ((4, 70, 60), {}),
    ((64, 61), {"two_d": True}), ((30, 257), {"two_d": True, "pml": (0, 0, 1, 1, 1, 0)}),
    ((250, 90), {"two_d": True, "K": 3, "L": 0}), ((33, 40), {"two_d": True, "batch": 2}),
    ((700, 250), {"two_d": True}),  # FP64: two rows per march
    ((690, 253), {"two_d": True}),  # FP64: and one row in the last
]


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("case", range(len(CASES)))
def test_direct_kernel_equals_marching_kernel(case, precision):
    room, kw = CASES[case]
    a = _solve(room, precision, 0, **kw)
    b = _solve(room, precision, 5, **kw)
    for x, y in zip(a, b):
        assert np.isfinite(x).all() and np.abs(a[0]).max() > 0
        assert np.array_equal(x, y)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("depth", [0, 3])  # the direct and the marching kernel
def test_samples_of_a_run_equal_those_of_single_steps(depth, precision):
    """A run records the samples of all but its last step in the stage launch that follows, and
    advances the step counter once (per graph, and per 16 steps beyond); single steps record each
    by the receiver kernel. Lengths around the graph (10) and the direct sequence (16); the source
    waveform follows the step either way."""
    h, c, rho, steps = 0.05, 343.0, 1.2, 47
    rng = np.random.default_rng(8)
    dt = 0.5 * h / c
    sc = scenes.box_room((33, 21, 17), h)
    m = mats.pack([mats.random_passive(rng, dt, c / (4 * h)) for _ in range(6)])

    def solve(parts):
        s = Solver(params(h=h, c=c, rho=rho, dt=dt, precision=precision))
        s.load_geometry(sc.S, sc.oid)
        s.set_materials(m["Rinf"], m["A"], m["zeta"], m["B"], m["Cc"], m["alpha"], m["beta"])
        s.set_sources(np.array([[12, 11, 10]], np.int32), np.array([1e-3]), 0, u_s=np.sin(0.3 * np.arange(2 * steps + 3)))
        s.set_receivers(np.array([[15, 11, 10], [30, 18, 5]], np.int32), steps)
        if depth:
            s.set_kz_chunk(depth)
        for n in parts:
            s.run(n)
        assert s.steps_done() == steps
        out = s.ir(), s.vel()
        s.close()
        return out

    one = solve([1] * steps)
    for parts in ([steps], [9, 10, 11, 17], [2, 45]):
        for x, y in zip(one, solve(parts)):
            assert np.array_equal(x, y)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("room,batch", [((9, 5, 4), 1), ((31, 17, 6), 3), ((140, 131, 117), 1), ((90, 80, 75), 4)])
def test_fields_come_back_as_they_were_set(room, batch, precision):
    """fz_get_fields packs the fields on the device: all at once while they are small (4 MB), else slabs
    of one field's rows, which may cross members."""
    sc = scenes.box_room(room, 0.05)
    s = Solver(params(h=0.05, precision=precision, batch=batch))
    s.load_geometry(sc.S, sc.oid)
    rng = np.random.default_rng(3)
    shape = ((batch,) if batch > 1 else ()) + sc.shape
    f = [rng.standard_normal(shape) for _ in range(4)]
    s.set_fields(*f)
    for got, want in zip(s.fields(), f):
        assert np.array_equal(got, want.astype(np.float32) if precision == "fp32" else want)
    s.close()
