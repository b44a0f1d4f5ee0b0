"""Performance cases of the stepper: what a user's program has it do, from the smallest solve to the largest.

A pass is a call sequence of the public API: `Solver.run` and the read-back of its receiver traces (a 3D room, a
planar room, a batch of sources over one room, a group of rooms), one evaluation of the misfit with its gradients
(`autograd.misfit` and `backward`), or one run of the 2D legacy scheme. Inputs are synthetic and made from the
seed: shoebox rooms with box obstacles, passive ADE wall materials, point sources, a Gaussian pulse, receivers.

`exact` is the same solve as plain torch operations in 64 bits.
"""
import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from fases_b200 import Group, Solver, params
from fases_b200.autograd import Room, misfit
from fases_b200.legacy2d import Legacy2D, plane_wave_fields, rect_scene

GHOST = 3
C0, RHO = 343.0, 1.2


# ---------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------
def _room(name, nx, ny, nz, steps, precision="fp32", batch=1, K=2, L=2, pml="001000", pml_cells=20, obstacles=3,
          h=0.02, tune=False, fields=False):
    return dict(name=name, kind="room", nx=nx, ny=ny, nz=nz, steps=steps, precision=precision, batch=batch, K=K, L=L,
                pml=pml, pml_cells=pml_cells, obstacles=obstacles, h=h, tune=tune, fields=fields)


def listed():
    return [
        # a test-sized room, run from a script that looks at the fields after a few steps: launches and latency
        _room("room_26x22x18_fp32", 26, 22, 18, 64, pml_cells=6, obstacles=1, h=0.05, fields=True),
        # the same kind of room in double precision, the arithmetic parity checks and fits use
        _room("room_45x38x29_fp64", 45, 38, 29, 64, precision="fp64", pml_cells=6, obstacles=1, h=0.05, fields=True),
        # a small project with measured wall materials of many poles (5 real, 3 pairs) and two open faces
        _room("room_71x53x47_poles_fp32", 71, 53, 47, 200, K=5, L=3, pml="001001", pml_cells=8, obstacles=2,
              h=0.04, fields=True),
        # a living room at audio bandwidth below 1 kHz, odd sizes, closed
        _room("room_119x103x87_fp32", 119, 103, 87, 200, pml="000000", tune=True),
        # a medium room, 7 M cells, one open face
        _room("room_192x192x192_fp32", 192, 192, 192, 100, tune=True),
        # the headline room: 10 x 8 x 4 m at h = 0.02 m, 40 M cells
        _room("room_500x400x200_fp32", 500, 400, 200, 60, obstacles=5, tune=True),
        # a precision study: the all-FP64 solve of a room of 4 M cells
        _room("room_190x150x140_fp64", 190, 150, 140, 40, precision="fp64", tune=True),
        # the planar FP64 solve (256 x 256 cells, 16-cell cPML)
        dict(name="plane_256x256_fp64", kind="plane", nx=256, ny=256, steps=200, precision="fp64", K=2, L=1,
             pml="001000", pml_cells=16, h=0.02, fields=True),
        # auralization: the responses to 12 source positions in one room, solved together
        _room("batch_12_of_96x84x70_fp32", 96, 84, 70, 60, batch=12, pml_cells=12),
        # a study of six rooms of different sizes stepped together
        dict(name="group_6_rooms_fp32", kind="group", rooms=6, lo=64, hi=160, steps=60, precision="fp32", K=2, L=2,
             pml="001000", pml_cells=20, obstacles=2, h=0.02),
        # one step of a material fit: the misfit of the responses and its gradient with respect to every wall
        # coefficient, in double precision (the scheme's |beta0 - beta2| has kinks: a gradient in 32 bits says
        # little past three digits)
        dict(name="gradient_78x66x54_fp64", kind="gradient", nx=78, ny=66, nz=54, steps=60, segment=30,
             precision="fp64", K=2, L=2, pml="001000", pml_cells=10, obstacles=1, h=0.04),
        # the 2D legacy scheme on a grid of the size its shipped project has
        dict(name="legacy2d_803x815_fp32", kind="legacy2d", nx=803, ny=815, steps=400, precision="fp32"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the listed ranges: rooms from 10^4 to 4 10^7 cells with aspect ratios up to about 2, odd sizes,
    closed or with one to three open faces, few or many poles, either precision."""
    kind = rng.choice(["room"] * 6 + ["batch", "group", "plane", "plane", "gradient", "legacy2d"])
    pml = rng.choice(["000000", "001000", "001000", "100010", "011001"])
    K, L = rng.choice([(2, 2), (2, 2), (1, 1), (4, 3), (5, 3)])
    prec = rng.choice(["fp32", "fp32", "fp64"])

    def edges(cells):
        a, b = rng.uniform(0.7, 1.4), rng.uniform(0.7, 1.4)
        e = cells ** (1.0 / 3.0)
        return max(16, int(e * a)), max(16, int(e * b)), max(16, int(e / (a * b)))

    if kind == "legacy2d":
        return dict(kind="legacy2d", nx=_log_int(rng, 90, 1200), ny=_log_int(rng, 90, 1000), steps=rng.randint(100, 400),
                    precision=prec)
    if kind == "plane":
        return dict(kind="plane", nx=_log_int(rng, 60, 1400), ny=_log_int(rng, 60, 1400), steps=rng.randint(60, 200),
                    precision=prec, K=K, L=L, pml=rng.choice(["000000", "001000", "001100"]), pml_cells=16, h=0.02,
                    fields=False)
    if kind == "group":
        lo = rng.randint(30, 80)
        return dict(kind="group", rooms=rng.randint(2, 8), lo=lo, hi=2 * lo, steps=rng.randint(30, 60),
                    precision="fp32", K=K, L=L, pml=pml, pml_cells=12, obstacles=1, h=0.02)
    if kind == "gradient":
        nx, ny, nz = edges(_log_int(rng, 20000, 300000))
        return dict(kind="gradient", nx=nx, ny=ny, nz=nz, steps=rng.randint(20, 60), segment=rng.choice([15, 30, 60]),
                    precision="fp64", K=K, L=L, pml=pml, pml_cells=5, obstacles=1, h=0.04)
    if kind == "batch":
        nx, ny, nz = edges(_log_int(rng, 30000, 800000))
        c = _room("", nx, ny, nz, rng.randint(30, 60), precision=prec, batch=rng.randint(2, 12), K=K, L=L, pml=pml,
                  pml_cells=8)
        del c["name"]
        return c
    cells = _log_int(rng, 10000, 39000000)
    nx, ny, nz = edges(cells)
    big = cells > 500000
    if big and prec == "fp64":
        nx, ny, nz = edges(min(cells, 8000000))
    c = _room("", nx, ny, nz, 40 if cells > 5000000 else rng.randint(60, 200), precision=prec, K=K, L=L, pml=pml,
              pml_cells=20 if big else 5, obstacles=rng.randint(0, 4), h=rng.choice([0.02, 0.03, 0.05]), tune=big,
              fields=cells < 200000)
    del c["name"]
    return c


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _box_scene(room, h, boxes, planar=False):
    """Signed distance (positive in air, clipped at 8 h) and material ids (layer + 1 where 0 <= S <= 3 h, 255
    elsewhere) of a shoebox with solid boxes, on the padded grid [Nz, Ny, Nx]; layers: the walls, then the boxes."""
    dev = _device()
    n = [room[0] + 2 * GHOST, room[1] + 2 * GHOST, (1 if planar else room[2]) + 2 * GHOST]
    ax = [((torch.arange(m, device=dev, dtype=torch.float64) + 0.5) * h).float() for m in n]
    X, Y, Z = ax[0][None, None, :], ax[1][None, :, None], ax[2][:, None, None]
    axes = (X, Y) if planar else (X, Y, Z)
    lo = torch.tensor(GHOST * h, dtype=torch.float32, device=dev)
    hi = [torch.tensor((GHOST + room[a]) * h, dtype=torch.float32, device=dev) for a in range(len(axes))]
    shape = (n[2], n[1], n[0])
    S = torch.full(shape, float("inf"), device=dev)
    layer = torch.zeros(shape, dtype=torch.uint8, device=dev)
    for a, x in enumerate(axes):
        for side, d in enumerate((x - lo, hi[a] - x)):
            near = d < S
            layer = torch.where(near, torch.full_like(layer, 2 * a + side), layer)
            S = torch.where(near, d.expand(shape), S)
    out2 = sum(torch.clamp(torch.maximum(lo - x, x - hi[a]), min=0) ** 2 for a, x in enumerate(axes))
    S = torch.where(S > 0, S, -torch.sqrt(out2).expand(shape))
    for q, (b0, b1) in enumerate(boxes):
        d = [torch.maximum(lo + b0[a] * h - x, x - (lo + b1[a] * h)) for a, x in enumerate(axes)]
        ext = torch.sqrt(sum(torch.clamp(x, min=0) ** 2 for x in d))
        inner = d[0]
        for x in d[1:]:
            inner = torch.maximum(inner, x)
        d = (ext + torch.clamp(inner, max=0)).expand(shape)
        layer = torch.where(d < S, torch.full_like(layer, 2 * len(axes) + q), layer)
        S = torch.minimum(S, d)
    S = torch.clamp(S, -8 * h, 8 * h)
    sel = (S >= 0) & (S <= np.float32(3.0 * h))
    for a in range(3):
        ends = [slice(None)] * 3
        for e in (0, -1):
            ends[a] = e
            sel[tuple(ends)] = False
    oid = torch.where(sel, layer + 1, torch.full_like(layer, 255))
    return S.cpu().numpy(), oid.cpu().numpy()


def _materials(rng, walls, matched, boxes, K, L):
    """Passive wall materials of K real poles and L complex pairs, |R| < 1 by the sum of the poles' peaks; the
    walls behind an open face are matched (R = 0), the boxes rigid (R = 0.99)."""
    n = walls + boxes
    m = {k: np.zeros((n, K)) for k in ("A", "zeta")}
    m.update({k: np.zeros((n, L)) for k in ("B", "Cc", "alpha", "beta")})
    m["Rinf"] = np.full(n, 0.99)
    m["zeta"][:] = np.exp(rng.uniform(math.log(1e2), math.log(8e3), (n, K)))
    m["alpha"][:] = np.exp(rng.uniform(math.log(2e2), math.log(5e3), (n, L)))
    m["beta"][:] = rng.uniform(300.0, 6000.0, (n, L))
    share = 0.25 / (K + 2 * L)
    for w in range(walls):
        if w in matched:
            m["Rinf"][w] = 0.0
            continue
        m["Rinf"][w] = rng.uniform(0.3, 0.7)
        m["A"][w] = m["zeta"][w] * rng.uniform(-share, share, K)
        m["B"][w] = m["alpha"][w] * rng.uniform(-share, share, L)
        m["Cc"][w] = m["alpha"][w] * rng.uniform(-share, share, L)
    return m


def _waveform(nsteps, dt, f0):
    """A Ricker-like pulse sampled at half steps."""
    t = (np.arange(2 * nsteps + 3) * 0.5 * dt - 1.2 / f0) * math.pi * f0
    return (1.0 - 2.0 * t * t) * np.exp(-t * t)


def _solve_inputs(case, seed, room=None):
    rng = np.random.default_rng([int(seed), 7])
    planar = case["kind"] == "plane"
    room = room or ((case["nx"], case["ny"]) if planar else (case["nx"], case["ny"], case["nz"]))
    h = case["h"]
    dt = 0.5 * h / C0
    boxes = []
    for _ in range(case.get("obstacles", 0)):
        b0, b1 = [], []
        for n in room:
            s = max(3, int(rng.uniform(0.06, 0.16) * n))
            a = int(rng.integers(max(2, n // 5), max(3, n - n // 5 - s)))
            b0.append(a)
            b1.append(a + s)
        boxes.append((b0, b1))
    S, oid = _box_scene(room, h, boxes, planar)
    pml = tuple(int(x) for x in case["pml"])  # faces U D R L F B: z-hi z-lo x-hi x-lo y-hi y-lo
    behind = [5, 4, 1, 0, 3, 2]
    mats = _materials(rng, 2 * len(room), {behind[f] for f in range(6) if pml[f]}, len(boxes), case["K"], case["L"])

    def free(count, clear):
        got = []
        for _ in range(20000):
            c = [int(rng.integers(GHOST + min(4, n // 4), GHOST + n - min(4, n // 4))) for n in room]
            c += [GHOST] * (3 - len(c))
            if S[c[2], c[1], c[0]] >= clear * h:
                got.append(c)
                if len(got) == count:
                    break
        return np.array(got, np.int32)

    batch = case.get("batch", 1)
    sources = free(batch if batch > 1 else 3, 3.5)
    receivers = free(16, 2.5)
    steps = case["steps"]
    out = dict(S=S, oid=oid, h=h, dt=dt, pml=pml, pml_cells=case["pml_cells"], mats=mats, src=sources, rec=receivers,
               planar=planar, sval=rng.uniform(5e-4, 1.5e-3, len(sources)), batch=batch,
               us=_waveform(4 * steps, dt, 0.1 * C0 / h), steps=steps)
    p0 = None
    if batch == 1:
        shape = S.shape
        p0 = np.zeros(shape)
        ctr = free(1, 4.5)[0] if min(room) > 12 else sources[0]
        r = 12
        sl, r2 = [], 0.0
        for a, m in ((2, shape[0]), (1, shape[1]), (0, shape[2])):
            i0, i1 = max(0, ctr[a] - r), min(m, ctr[a] + r + 1)
            if planar and a == 2:
                i0, i1 = GHOST, GHOST + 1
            sl.append(slice(i0, i1))
            x = (np.arange(i0, i1) - ctr[a]).astype(float) ** 2
            r2 = r2 + x.reshape([-1 if q == 2 - a else 1 for q in range(3)])
        p0[tuple(sl)] = np.exp(-r2 / 8.0) * (S[tuple(sl)] >= np.float32(h))
    out["p0"] = p0
    return out


def _legacy_inputs(case, seed):
    rng = np.random.default_rng([int(seed), 11])
    nx, ny = case["nx"], case["ny"]
    h = float(np.float32(0.005))
    wx, wy = nx * h, ny * h
    rects = []
    for layer in (1, 2):
        x0, y0 = rng.uniform(0.35, 0.55) * wx, rng.uniform(0.15, 0.5) * wy
        rects.append(((x0, y0), (x0 + rng.uniform(0.05, 0.2) * wx, y0 + rng.uniform(0.1, 0.35) * wy), layer))
    rects += [((0.0, 0.0), (wx, 8 * h), 1)]  # a floor
    S, oid = rect_scene(nx, ny, h, rects)
    mats = _materials(rng, 2, set(), 0, 2, 1)
    src_x = float(rng.uniform(0.15, 0.25) * wx)
    return dict(S=S, oid=oid, mats=mats, src_x=src_x, rec=(int(src_x / h) + 10, ny - ny // 4), steps=case["steps"])


def _set_up(s, d, capacity):
    m = d["mats"]
    s.load_geometry(d["S"], d["oid"])
    s.set_materials(m["Rinf"], m["A"], m["zeta"], m["B"], m["Cc"], m["alpha"], m["beta"])
    s.set_sources(d["src"], d["sval"], 0, u_s=d["us"])
    if d["batch"] > 1:
        s.set_source_members(np.arange(d["batch"]))
    s.set_receivers(d["rec"], capacity)
    if d["p0"] is not None:
        s.set_fields(p=d["p0"])


def _solver(case, d):
    s = Solver(params(h=d["h"], c=C0, rho=RHO, dt=d["dt"], pml=d["pml"], pml_cells=d["pml_cells"],
                      precision=case["precision"], two_d=d["planar"], batch=d["batch"]))
    # traces of a job of several passes
    _set_up(s, d, 4 * d["steps"])
    return s


def _group_rooms(case, seed):
    rng = np.random.default_rng([int(seed), 3])
    return [tuple(int(x) for x in rng.integers(case["lo"], case["hi"] + 1, 3)) for _ in range(case["rooms"])]


def _target(d, seed):
    """Measured-looking responses: decaying noise of about the traces' level."""
    rng = np.random.default_rng([int(seed), 5])
    t = np.arange(d["steps"])
    return 0.05 * rng.standard_normal((len(d["rec"]), d["steps"])) * np.exp(-t / d["steps"])


def _theta(m):
    return np.concatenate([m["Rinf"][:, None]] + [m[k] for k in ("A", "zeta", "B", "Cc", "alpha", "beta")], axis=1)


def prepare(case, seed):
    if case["kind"] == "legacy2d":
        d = _legacy_inputs(case, seed)
        s = Legacy2D(case["nx"], case["ny"], precision=case["precision"])
        m = d["mats"]
        s.load_geometry(d["S"], d["oid"])
        s.set_materials(m["Rinf"], m["A"], m["zeta"], m["B"], m["Cc"], m["alpha"], m["beta"])
        q = s.params
        s.set_receiver(d["rec"][0], d["rec"][1], d["steps"])
        start = plane_wave_fields(case["nx"], case["ny"], q.h, d["src_x"], q.rho, q.c)
        return {"case": case, "solver": s, "start": start}
    if case["kind"] == "gradient":
        d = _solve_inputs(case, seed)
        prm = dict(h=d["h"], c=C0, rho=RHO, dt=d["dt"], pml=d["pml"], pml_cells=d["pml_cells"],
                   precision=case["precision"])
        room = Room(d["S"], d["oid"], prm, d["rec"], d["steps"], _theta(d["mats"]), src_cells=d["src"],
                    sval0=d["sval"], u_s=d["us"], p0=d["p0"], K=case["K"], L=case["L"], segment_steps=case["segment"])
        theta = torch.tensor(room.materials0, requires_grad=True)
        return {"case": case, "room": room, "target": torch.tensor(_target(d, seed)), "theta": theta}
    if case["kind"] == "group":
        members = [_solver(case, _solve_inputs(case, 1000 * int(seed) + q, r))
                   for q, r in enumerate(_group_rooms(case, seed))]
        g = Group(members)
        g.autotune()
        return {"case": case, "group": g, "members": members}
    s = _solver(case, _solve_inputs(case, seed))
    if case.get("tune"):
        s.autotune()  # as the command line does for runs of this length
    s.prepare()
    return {"case": case, "solver": s}


# ---------------------------------------------------------------------------------------------
# a pass
# ---------------------------------------------------------------------------------------------
def _traces(s, case):
    # an FP32 solve's traces as the 32-bit samples of the IR file, an FP64 solve's in full
    return {"ir": s.ir(fp64=case["precision"] == "fp64"), "vel": s.vel()}


def run(state):
    case = state["case"]
    if case["kind"] == "legacy2d":
        # one response: the incoming wave set, the steps, the trace
        s = state["solver"]
        s.set_fields(*state["start"])
        s.run(case["steps"])
        ir, f = s.ir(), s.fields()
        if case["precision"] == "fp32":
            ir, f = ir.astype(np.float32), [x.astype(np.float32) for x in f]
        return {"ir": ir, "fields": f}
    if case["kind"] == "gradient":
        theta = state["theta"]
        theta.grad = None
        J = misfit(state["room"], state["target"], theta)
        J.backward()
        return {"J": J.detach(), "theta": theta.grad}
    if case["kind"] == "group":
        state["group"].run(case["steps"])
        return [_traces(s, case) for s in state["members"]]
    s = state["solver"]
    s.run(case["steps"])
    out = _traces(s, case)
    if case["fields"]:
        f = s.fields()
        out["fields"] = f if case["precision"] == "fp64" else [x.astype(np.float32) for x in f]
    return out


def _room_work(cells, band, steps, precision, K, L):
    """A step reads and writes the state once (p, u, v, w; at the band the pole states, 64 bits); each of its three
    stages reconstructs two variables at two faces in three directions (about 60 operations a variable and
    direction) and combines them (about 50), a band cell interpolates and steps its poles (about 100)."""
    b = 4 if precision == "fp32" else 8
    return {"bytes": steps * (cells * 8.0 * b + band * (K + 2 * L) * 16.0),
            "flops": steps * 3.0 * (cells * (3 * 2 * 60.0 + 50.0) + band * (100.0 + 8 * K + 16 * L))}


def work(case):
    if case["kind"] == "legacy2d":
        n = (case["nx"] - 6.0) * (case["ny"] - 6.0) * case["steps"]
        b = 4 if case["precision"] == "fp32" else 8
        return {"bytes": n * 6 * b, "flops": n * 3 * (2 * 2 * 70.0 + 40.0)}
    if case["kind"] == "plane":
        cells = float(case["nx"] * case["ny"])
        b = 4 if case["precision"] == "fp32" else 8
        return {"bytes": case["steps"] * cells * 6.0 * b, "flops": case["steps"] * 3 * cells * (2 * 2 * 60.0 + 40.0)}
    if case["kind"] == "group":
        e = 0.5 * (case["lo"] + case["hi"])
        w = _room_work(e ** 3, 18 * e * e, case["steps"], case["precision"], case["K"], case["L"])
        return {k: v * case["rooms"] for k, v in w.items()}
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    band = 6.0 * (nx * ny + ny * nz + nx * nz)
    w = _room_work(float(nx * ny * nz), band, case["steps"], case["precision"], case["K"], case["L"])
    # the gradient: the forward pass, and the reverse pass at about twice its operations
    times = 3.0 if case["kind"] == "gradient" else float(case.get("batch", 1))
    return {k: v * times for k, v in w.items()}


# ---------------------------------------------------------------------------------------------
# the same solves as plain torch in 64 bits
# ---------------------------------------------------------------------------------------------
def _at(q, dim, lo, n):
    return q.narrow(dim, lo, n)


def _weno_z(q, dim):
    """(V-(i+1/2), V+(i-1/2)) of the centres i = 2 .. N-3 along dim."""
    n = q.shape[dim] - 4
    m2, m1, c, p1, p2 = (_at(q, dim, o, n) for o in range(5))
    beta = [13.0 / 12.0 * (c - 2 * p1 + p2) ** 2 + 0.25 * (3 * c - 4 * p1 + p2) ** 2,
            13.0 / 12.0 * (m1 - 2 * c + p1) ** 2 + 0.25 * (m1 - p1) ** 2,
            13.0 / 12.0 * (m2 - 2 * m1 + c) ** 2 + 0.25 * (m2 - 4 * m1 + 3 * c) ** 2]
    tau = (beta[0] - beta[2]).abs()
    z = [1.0 + tau / (b + 1e-10) for b in beta]
    lo = [(2 * c + 5 * p1 - p2) / 6, (-m1 + 5 * c + 2 * p1) / 6, (2 * m2 - 7 * m1 + 11 * c) / 6]
    hi = [(11 * c - 7 * p1 + 2 * p2) / 6, (2 * m1 + 5 * c - p1) / 6, (-m2 + 5 * m1 + 2 * c) / 6]
    out = []
    for cand, d in ((lo, (0.3, 0.6, 0.1)), (hi, (0.1, 0.6, 0.3))):
        a = [d[r] * z[r] for r in range(3)]
        out.append((a[0] * cand[0] + a[1] * cand[1] + a[2] * cand[2]) / (a[0] + a[1] + a[2]))
    return out


def _flux_difference(p, q, dim, h):
    """(-dF_p, -dF_q) / h of the interior cells 3 .. N-4 along dim (exact Riemann flux of linear acoustics)."""
    (pm, pp), (qm, qp) = _weno_z(p, dim), _weno_z(q, dim)
    n = pm.shape[dim] - 1  # faces between centres 2 .. N-3
    pl, pr, ql, qr = _at(pm, dim, 0, n), _at(pp, dim, 1, n), _at(qm, dim, 0, n), _at(qp, dim, 1, n)
    fp = 0.5 * (RHO * C0 * C0 * (qr + ql) - C0 * (pr - pl))
    fq = 0.5 * ((pr + pl) / RHO - C0 * (qr - ql))
    return [(_at(f, dim, 0, n - 1) - _at(f, dim, 1, n - 1)) / h for f in (fp, fq)]


class _Exact:
    """One solve: fields [Nz, Ny, Nx] of three rotating sets, pole states per band cell."""

    def __init__(self, d, theta=None, member=None):
        dev = _device()
        f64 = dict(dtype=torch.float64, device=dev)
        self.d, self.h, self.dt, self.planar = d, d["h"], d["dt"], d["planar"]
        S = torch.as_tensor(d["S"], device=dev)
        self.shape = S.shape
        Nz, Ny, Nx = S.shape
        inner = torch.zeros(S.shape, dtype=torch.bool, device=dev)
        inner[3:-3, 3:-3, 3:-3] = True
        self.update = inner & ~(S < np.float32(self.h))
        oid = torch.as_tensor(d["oid"], device=dev)
        band = inner & (oid != 0) & (oid != 255)
        self.b = band.reshape(-1).nonzero().reshape(-1)
        k, j, i = (x.reshape(-1) for x in torch.nonzero(band, as_tuple=True))
        S = S.to(torch.float64)
        g = torch.stack([(S[k, j, i + 1] - S[k, j, i - 1]), (S[k, j + 1, i] - S[k, j - 1, i]),
                         (S[k + 1, j, i] - S[k - 1, j, i])]) * (0.5 / self.h)
        self.n = -g / torch.clamp(torch.sqrt((g * g).sum(0)), min=1e-12)
        s = S[k, j, i]
        foot = torch.stack([i, j, k]).to(torch.float64) - 2.0 * self.n  # C - 2 h n in cells
        top = torch.tensor([Nx - 2, Ny - 2, Nz - 2], device=dev)[:, None]
        base = torch.minimum(torch.clamp(torch.floor(foot + 1e-12), min=0), top)
        fr = foot - base
        base = base.long()
        self.corners = []
        for c in range(8):
            o = (c & 1, (c >> 1) & 1, c >> 2)
            at = (base[0] + o[0]) + Nx * ((base[1] + o[1]) + Ny * (base[2] + o[2]))
            w = 1.0
            for a in range(3):
                w = w * (fr[a] if o[a] else 1.0 - fr[a])
            self.corners.append((at, w))
        tol = 3.0 * self.h
        r = (s - self.h) / (tol - self.h)
        self.chi = torch.where(s >= tol, torch.zeros_like(s),
                               torch.where(s <= self.h, torch.ones_like(s), 1.0 - r * r * (3.0 - 2.0 * r)))
        self.mat = oid[k, j, i].long() - 1
        m = d["mats"]
        self.K, self.L = m["A"].shape[1], m["B"].shape[1]
        self.theta = theta if theta is not None else torch.as_tensor(_theta(m), **f64)
        self.sval = torch.as_tensor(d["sval"], **f64)
        use = range(len(d["src"])) if member is None else [member]
        self.src = [(q, int(c[0] + Nx * (c[1] + Ny * c[2]))) for q, c in enumerate(d["src"]) if q in use]
        self.us = d["us"]
        rc = np.asarray(d["rec"])
        self.rec = torch.as_tensor(rc[:, 0] + Nx * (rc[:, 1] + Ny * rc[:, 2]), device=dev).long()
        zero = torch.zeros(S.shape, **f64)
        first = zero if d["p0"] is None else torch.as_tensor(d["p0"], **f64)
        self.U0 = [first, zero, zero, zero]
        self.U1 = [zero] * 4
        self.U2 = [zero] * 4
        nb = len(self.b)
        self.poles = [torch.zeros((nb, x), **f64) for x in (self.K, self.L, self.L)]
        # cPML profiles along x, y, z on the interior cells
        self.pml, self.psi = [None] * 3, [None] * 3
        faces = d["pml"]
        nd = d["pml_cells"]
        for a, (N, lo, hi) in enumerate(((Nx, faces[3], faces[2]), (Ny, faces[5], faces[4]), (Nz, faces[1], faces[0]))):
            if not (lo or hi):
                continue
            x = np.arange(3, N - 3).astype(float)
            xm, xp = np.clip((3 + nd - x) / nd, 0, 1), np.clip((x - (N - 4 - nd)) / nd, 0, 1)
            pref = 0.5 * C0 * 3.0 * math.log(1e7) / (nd * self.h)
            sig = pref * (lo * xm ** 2 + hi * xp ** 2)
            dep = lo * xm + hi * xp
            kap = 1.0 + 4.0 * dep ** 2
            amax = 20.0 * math.pi
            alp = 0.1 * amax + 0.9 * amax * (1.0 - dep)
            bb = np.exp(-(alp + sig / kap) * self.dt)
            ca = np.where(sig > 0, sig / (kap * (sig + kap * alp)) * (bb - 1.0), 0.0)
            inside = ((x < 3 + nd) & bool(lo)) | ((x >= N - 3 - nd) & bool(hi))
            sh = [1, 1, 1]
            sh[2 - a] = -1
            self.pml[a] = [torch.as_tensor(np.where(inside, v, 0.0), **f64).reshape(sh)
                           for v in (1.0 / kap - 1.0, bb, ca, np.ones_like(kap))]
            self.psi[a] = [zero[3:-3, 3:-3, 3:-3]] * 2

    def stage(self, st, U, base, old, psi):
        """Fields after stage st's update, cPML and sources, and the cPML states (advanced in stage 2)."""
        p = U[0]
        cut = [slice(3, -3)] * 3
        D = []
        for a in range(3):
            if a == 2 and self.planar:
                D.append([torch.zeros_like(D[0][0])] * 2)
                continue
            win = list(cut)
            win[2 - a] = slice(None)
            D.append(_flux_difference(p[tuple(win)], U[1 + a][tuple(win)], 2 - a, self.h))
        rate = [D[0][0] + D[1][0] + D[2][0], D[0][1], D[1][1], D[2][1]]
        c = tuple(cut)
        new = []
        for f in range(4):
            x = U[f][c] + self.dt * rate[f]
            x = x if st == 0 else 0.75 * base[f][c] + 0.25 * x if st == 1 else (base[f][c] + 2.0 * x) / 3.0
            new.append(x)
        w = (1.0, 0.25, 2.0 / 3.0)[st] * self.dt
        upd = self.update[c]
        out_psi = list(psi)
        for a in range(3):
            if self.pml[a] is None:
                continue
            k1, b, ca, ins = self.pml[a]
            for q, f in ((0, 0), (1, 1 + a)):
                new[f] = new[f] + w * (k1 * D[a][q] + ins * psi[a][q])
            if st == 2:
                out_psi[a] = [torch.where(upd, b * psi[a][q] + ca * D[a][q], psi[a][q]) for q in (0, 1)]
        out = []
        for f in range(4):
            x = torch.where(upd, new[f], old[f][c])
            x = torch.nn.functional.pad(x, (3,) * 6)
            rim = old[f].clone()
            rim[c] = 0.0
            out.append(x + rim)
        return out, out_psi

    def inject(self, p, st, n):
        nn = 2 * n + (0, 2, 1)[st]
        if nn >= len(self.us):
            return p
        unit = (1.0, 0.25, 2.0 / 3.0)[st] * self.dt * C0 * C0 * RHO * 6.0 / self.h * self.us[nn]
        flat = p.reshape(-1)
        for q, at in self.src:
            flat = flat.index_add(0, torch.tensor([at], device=p.device), (self.sval[q] * unit).reshape(1))
        return flat.reshape(self.shape)

    def boundary(self, st, U, out, mid, right):
        """The band cells' blend, and the pole states after the stage."""
        D = [sum(w * u.reshape(-1)[at] for at, w in self.corners) for u in U]
        n = self.n
        un = D[1] * n[0] + D[2] * n[1] + D[3] * n[2]
        Z0 = RHO * C0
        wout = D[0] + Z0 * un
        t = self.theta[self.mat]
        K, L = self.K, self.L
        R, A, zeta = t[:, 0], t[:, 1:1 + K], t[:, 1 + K:1 + 2 * K]
        B, Cc, al, be = (t[:, 1 + 2 * K + q * L:1 + 2 * K + (q + 1) * L] for q in range(4))
        a_, b_, c_ = ((0.0, 1.0, 1.0), (3.0, 1.0, 4.0), (1.0, 2.0, 3.0))[st]
        wo = wout[:, None]
        rate = [wo - zeta * right[0], wo - (al * right[1] + be * right[2]), be * right[1] - al * right[2]]
        new = [(a_ * m + b_ * (r + self.dt * x)) / c_ for m, r, x in zip(mid, right, rate)]
        win = R * wout + (A * new[0]).sum(1) + (B * new[1]).sum(1) + (Cc * new[2]).sum(1)
        pb, unb = 0.5 * (win + wout), (wout - win) / (2.0 * Z0)
        val = [pb] + [unb * n[a] + (D[1 + a] - un * n[a]) for a in range(3)]
        res = []
        for f in range(4):
            flat = out[f].reshape(-1)
            res.append(flat.index_put((self.b,), (1.0 - self.chi) * flat[self.b] + self.chi * val[f])
                       .reshape(self.shape))
        return res, new

    def _step(self, n, U0, U1, U2, poles, psi):
        x, psi = self.stage(0, U0, U0, U1, psi)
        x[0] = self.inject(x[0], 0, n)
        x1, s1 = self.boundary(0, U0, x, poles, poles)
        x, psi = self.stage(1, x1, U0, U2, psi)
        x[0] = self.inject(x[0], 1, n)
        x2, s2 = self.boundary(1, x1, x, poles, s1)
        x, psi = self.stage(2, x2, U0, x1, psi)
        x[0] = self.inject(x[0], 2, n)
        x3, s3 = self.boundary(2, x2, x, poles, s2)
        return x3, x2, s3, psi

    def step(self, n):
        new, U2, poles, psi = self._step(n, self.U0, self.U1, self.U2, self.poles, self.psi)
        self.U0, self.U1, self.U2, self.poles, self.psi = new, self.U0, U2, poles, psi

    def samples(self):
        return torch.stack([f.reshape(-1)[self.rec] for f in self.U0])  # [4, n_rec]

    def solve(self, steps):
        got = []
        with torch.no_grad():
            for n in range(steps):
                self.step(n)
                got.append(self.samples())
        t = torch.stack(got)  # [steps, 4, n_rec]
        return t[:, 0].t().cpu().numpy().copy(), t[:, 1:].permute(2, 0, 1).cpu().numpy().copy()


def _exact_room(d, steps, fields):
    if d["batch"] > 1:
        both = [_Exact(d, member=m).solve(steps) for m in range(d["batch"])]
        return {"ir": np.stack([x[0] for x in both]), "vel": np.stack([x[1] for x in both])}
    e = _Exact(d)
    ir, vel = e.solve(steps)
    out = {"ir": ir, "vel": vel}
    if fields:
        out["fields"] = [f.cpu().numpy() for f in e.U0]
    return out


def _exact_gradient(case, d, seed):
    dev = _device()
    theta = torch.tensor(_theta(d["mats"]), dtype=torch.float64, device=dev, requires_grad=True)
    e = _Exact(d, theta)
    target = torch.as_tensor(_target(d, seed), device=dev)
    J = 0.0
    flat = lambda: [*e.U0, *e.U1, *e.U2, *e.poles, *[q for a in e.psi if a for q in a]]  # noqa: E731

    def one(n, *v):
        ps, at = [], 15
        for a in e.psi:
            ps.append(list(v[at:at + 2]) if a else None)
            at += 2 if a else 0
        new, U2, poles, psi = e._step(n, list(v[0:4]), list(v[4:8]), list(v[8:12]), list(v[12:15]), ps)
        return (*new, *v[0:4], *U2, *poles, *[q for a in psi if a for q in a])

    for n in range(d["steps"]):
        v = checkpoint(one, n, *flat(), use_reentrant=False)
        e.U0, e.U1, e.U2, e.poles = list(v[0:4]), list(v[4:8]), list(v[8:12]), list(v[12:15])
        at = 15
        for a in range(3):
            if e.psi[a]:
                e.psi[a] = list(v[at:at + 2])
                at += 2
        J = J + ((e.U0[0].reshape(-1)[e.rec] - target[:, n]) ** 2).sum()
    J.backward()
    return {"J": J.detach().cpu(), "theta": theta.grad.cpu()}


def _weno_js(q, dim, eps):
    n = q.shape[dim] - 4
    m2, m1, c, p1, p2 = (_at(q, dim, o, n) for o in range(5))
    beta = [13.0 / 12.0 * (c - 2 * p1 + p2) ** 2 + 0.25 * (3 * c - 4 * p1 + p2) ** 2,
            13.0 / 12.0 * (m1 - 2 * c + p1) ** 2 + 0.25 * (m1 - p1) ** 2,
            13.0 / 12.0 * (m2 - 2 * m1 + c) ** 2 + 0.25 * (m2 - 4 * m1 + 3 * c) ** 2]
    lo = [(2 * c + 5 * p1 - p2) / 6, (-m1 + 5 * c + 2 * p1) / 6, (2 * m2 - 7 * m1 + 11 * c) / 6]
    hi = [(11 * c - 7 * p1 + 2 * p2) / 6, (2 * m1 + 5 * c - p1) / 6, (-m2 + 5 * m1 + 2 * c) / 6]
    out = []
    for cand, w in ((lo, (0.3, 0.6, 0.1)), (hi, (0.1, 0.6, 0.3))):
        a = [w[r] / (beta[r] + eps) ** 2 for r in range(3)]
        out.append((a[0] * cand[0] + a[1] * cand[1] + a[2] * cand[2]) / (a[0] + a[1] + a[2]))
    return out


def _exact_legacy(case, d):
    dev = _device()
    nx, ny = case["nx"], case["ny"]
    f32 = np.float32
    h = float(f32(0.005))
    c = float(np.sqrt(f32(1.4) * f32(287.05) * f32(f32(22.0) + f32(273.15)), dtype=f32))
    rho, eps, tol = float(f32(1.225)), float(f32(1e-7)), float(f32(3.0) * f32(0.005))
    dt = float(f32(f32(0.2) * f32(0.005) / f32(c)))
    f64 = dict(dtype=torch.float64, device=dev)
    S32 = torch.as_tensor(d["S"], device=dev)
    S = S32.to(torch.float64)
    oid = torch.as_tensor(d["oid"], device=dev)
    inner = torch.zeros((ny, nx), dtype=torch.bool, device=dev)
    inner[3:-3, 3:-3] = True
    fluid = inner & ~(S32 < f32(h))
    band = inner & (oid != 0) & (oid != 255)
    j, i = torch.nonzero(band, as_tuple=True)
    s = S[j, i]
    g = torch.stack([S[j, i + 1] - S[j, i - 1], S[j + 1, i] - S[j - 1, i]]) * (0.5 / h)
    nrm = -g / torch.clamp(torch.sqrt((g * g).sum(0)), min=1e-12)
    foot = torch.stack([i, j]).to(torch.float64) - nrm
    base = torch.floor(foot + 1e-6)
    fr = foot - base
    base = base.long()
    r = (s - h) / (tol - h)
    chi = torch.where(s >= tol, torch.zeros_like(s),
                      torch.where(s <= h, torch.ones_like(s), 1.0 - r * r * (3.0 - 2.0 * r)))
    cub = lambda t: (-t * (t - 2) * (t - 1) / 6, (t - 2) * (t - 1) * (t + 1) / 2,  # noqa: E731
                     t * (-t * t + t + 2) / 2, t * (t * t - 1) / 6)
    wx, wy = cub(fr[0]), cub(fr[1])
    m = {k: torch.as_tensor(v, **f64) for k, v in d["mats"].items()}
    mat = oid[j, i].long() - 1
    half = float(int(f32(0.15) * f32(min(nx, ny))))
    ly = torch.clamp((half - torch.arange(ny, **f64)) / half, 0, 1)
    uy = torch.clamp((torch.arange(ny, **f64) - (ny - half)) / half, 0, 1)
    sp = torch.clamp(float(f32(0.018)) * (ly ** 3 + uy ** 3), max=float(f32(0.999)))[:, None]  # absorbing y faces
    colfluid = fluid.any(0)
    zero = torch.zeros((ny, nx), **f64)
    p0 = plane_wave_fields(nx, ny, h, d["src_x"], rho, c)
    U0 = [torch.as_tensor(x, **f64).to(torch.float32 if case["precision"] == "fp32" else torch.float64).to(torch.float64)
          for x in p0]
    U1, U2 = [zero.clone() for _ in range(3)], [zero.clone() for _ in range(3)]
    nb = len(j)
    poles = [torch.zeros((nb, x), **f64) for x in (m["A"].shape[1], m["B"].shape[1], m["B"].shape[1])]
    Z0 = rho * c

    def stage(st, U, out, mid, right):
        D = []
        for dim, f in ((1, 1), (0, 2)):
            win = (slice(3, -3), slice(None)) if dim == 1 else (slice(None), slice(3, -3))
            (pm, pp), (qm, qp) = _weno_js(U[0][win], dim, eps), _weno_js(U[f][win], dim, eps)
            n = pm.shape[dim] - 1
            pl, pr, ql, qr = _at(pm, dim, 0, n), _at(pp, dim, 1, n), _at(qm, dim, 0, n), _at(qp, dim, 1, n)
            fp = 0.5 * (rho * c * c * (qr + ql) - c * (pr - pl))
            fq = 0.5 * ((pr + pl) / rho - c * (qr - ql))
            D.append([(_at(x, dim, 0, n - 1) - _at(x, dim, 1, n - 1)) / h for x in (fp, fq)])
        rate = [D[0][0] + D[1][0], D[0][1], D[1][1]]
        cut = (slice(3, -3), slice(3, -3))
        new = []
        for f in range(3):
            x = U[f][cut] + dt * rate[f]
            x = x if st == 0 else 0.75 * U0[f][cut] + 0.25 * x if st == 1 else (U0[f][cut] + 2.0 * x) / 3.0
            x = x - sp[3:-3] * x
            y = out[f].clone()
            y[cut] = torch.where(fluid[cut], x, y[cut])
            new.append(y)
        for f in (0, 2):
            y = new[f]
            for rows, src in (((0, 1, 2), 3), ((ny - 3, ny - 2), ny - 4), ((ny - 1,), ny - 5)):
                for rr in rows:
                    y[rr, 3:-3] = torch.where(colfluid[3:-3], y[src, 3:-3], y[rr, 3:-3])
        P = []
        for f in range(3):
            acc = 0.0
            for b in range(4):
                for a in range(4):
                    acc = acc + wy[b] * wx[a] * U[f][base[1] + b - 1, base[0] + a - 1]
            P.append(acc)
        un, ut = P[1] * nrm[0] + P[2] * nrm[1], -P[1] * nrm[1] + P[2] * nrm[0]
        wout = P[0] + Z0 * un
        wo = wout[:, None]
        a_, b_, c_ = ((0.0, 1.0, 1.0), (3.0, 1.0, 4.0), (1.0, 2.0, 3.0))[st]
        al, be = m["alpha"][mat], m["beta"][mat]
        dr = [wo - m["zeta"][mat] * right[0], wo - (al * right[1] + be * right[2]), be * right[1] - al * right[2]]
        pol = [(a_ * x + b_ * (y + dt * z)) / c_ for x, y, z in zip(mid, right, dr)]
        win = (m["Rinf"][mat] * wout + (m["A"][mat] * pol[0]).sum(1) + (m["B"][mat] * pol[1]).sum(1)
               + (m["Cc"][mat] * pol[2]).sum(1))
        unb = (wout - win) / (2.0 * Z0)
        val = [0.5 * (win + wout), unb * nrm[0] - ut * nrm[1], unb * nrm[1] + ut * nrm[0]]
        for f in range(3):
            new[f][j, i] = (1.0 - chi) * new[f][j, i] + chi * val[f]
        return new, pol

    got = []
    for n in range(d["steps"]):
        U1, s1 = stage(0, U0, U1, poles, poles)
        U2, s2 = stage(1, U1, U2, poles, s1)
        U1, poles = stage(2, U2, U1, poles, s2)
        U0 = [x.clone() for x in U1]
        got.append(U0[0][d["rec"][1], d["rec"][0]])
    return {"ir": torch.stack(got).cpu().numpy(), "fields": [x.cpu().numpy() for x in U0]}


def exact(case, seed):
    kind = case["kind"]
    if kind == "legacy2d":
        return _exact_legacy(case, _legacy_inputs(case, seed))
    if kind == "group":
        cells = case["rooms"] * (0.5 * (case["lo"] + case["hi"])) ** 3
        if cells * case["steps"] > 7e8:
            return None
        return [_exact_room(_solve_inputs(case, 1000 * int(seed) + q, r), case["steps"], False)
                for q, r in enumerate(_group_rooms(case, seed))]
    cells = float(case["nx"] * case["ny"] * (7 if kind == "plane" else case["nz"])) * case.get("batch", 1)
    if cells * case["steps"] > 1e9:
        return None  # the largest take minutes
    d = _solve_inputs(case, seed)
    if kind == "gradient":
        return _exact_gradient(case, d, seed)
    return _exact_room(d, case["steps"], case["fields"])
