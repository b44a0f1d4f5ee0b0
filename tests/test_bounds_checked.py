"""The bounds-checked build (libfz_checked.so, compiled with -DFZ_BOUNDS_CHECK; loaded when
FZ_BOUNDS_CHECK=1): every computed global index of the stepping kernels (direct stage; marching stage and
band; receivers) and of the adjoint kernels is checked against its array, and an out-of-range one would
set an error bit (FZ_EBOUNDS at the next sync) instead of being accessed. compute-sanitizer is not
available for this purpose, so this build stands in for its memcheck. The same solves -- cPML on
every face, an obstacle band, PCS source, receivers; five real poles a wall; a batch of three; a planar
room; ragged tiles; FP32 and FP64 -- and a gradient with every output (materials, sources, cPML, initial
fields), each by the direct kernel and, with a tile depth set, by the marching and band kernels, and a
group with shared launches, run in a child process on the checked build must finish without an error and
reproduce the normal build's traces bit for bit (the gradient to 1e-5: its atomics sum in a varying
order)."""
import ctypes
import json
import os
import subprocess
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CHECKED = os.path.join(ROOT, "fases_b200", "libfz_checked.so")

SCRIPT = r'''
import json, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
from fases_b200 import Group, Solver, params, scenes
from fases_b200 import materials as mats
from tests.helpers import small_room, run_gpu
from tests import test_adjoint_params as ap
from tests import test_batch as tb
out = {"bands": {}}

def select(s, name, depth):
    # a depth that is not the heuristic one selects the marching kernel and its band launches
    if depth:
        s.set_kz_chunk(depth)
        s.profile(True)
        s.run(1)
        out["bands"][name] = s.profile_read()["band"][1]
        s.profile(False)

for depth in (0, 5):
    for name, kw, prec in [("box_all_pml", dict(seed=6, room=(30, 30, 30), pml=(1, 1, 1, 1, 1, 1), pml_cells=5, steps=25), "fp32"),
                           ("box_fp64", dict(seed=7, steps=25), "fp64"),
                           ("poles", dict(seed=9, K=5, L=3, steps=23), "fp32"),
                           ("ragged", dict(seed=8, room=(37, 21, 19), pml=(0, 1, 0, 1, 0, 1), pml_cells=4, steps=22), "fp32")]:
        cfg = small_room(**kw)
        s = run_gpu(cfg, prec, run=False)
        name += "/%d" % depth
        select(s, name, depth)
        s.run(kw["steps"] - (1 if depth else 0))
        s.sync()
        out[name] = s.ir().tolist()
        s.close()
    cfg = small_room(seed=11, pml=(1, 0, 1, 0, 0, 1), steps=21, pulse=False)
    b = tb._solver(cfg, "fp32", batch=3, members=np.arange(3))
    select(b, "batch/%d" % depth, depth)
    b.run(21 - (1 if depth else 0))
    out["batch/%d" % depth] = b.ir().tolist()
    b.close()
    sc = scenes.box_room_2d((95, 71), 0.05)
    s = Solver(params(h=0.05, precision="fp64", two_d=True, pml=(0, 0, 1, 0, 1, 0), pml_cells=6))
    s.load_geometry(sc.S, sc.oid)
    m = mats.pack([mats.rigid(0.9)] * 4)
    s.set_materials(m["Rinf"], m["A"], m["zeta"], m["B"], m["Cc"], m["alpha"], m["beta"])
    s.set_receivers(np.array([[40, 30, 3], [90, 70, 3]], np.int32), 24)
    s.set_fields(p=scenes.gaussian_pulse(sc.shape, 0.05, (50, 40, 3), 3.0, amplitude=0.5))
    select(s, "plane/%d" % depth, depth)
    s.run(24 - (1 if depth else 0))
    out["plane/%d" % depth] = s.ir().tolist()
    s.close()
    cfg = ap._cfg()
    tgt = ap._target(cfg)
    s = ap._solver(cfg, precision="fp32")
    if depth:
        s.set_kz_chunk(depth)
    g = s.misfit_gradient(tgt, segment_steps=16, sources=True, pml=True, initial=True)
    s.close()
    out["grad/%d" % depth] = [g["raw"].ravel().tolist(), g["sval"].tolist(),
                              [g["pml"][k] for k in ("R0", "kappa_max", "alpha_max")], g["initial"][0].ravel().tolist()]
cfgs = [small_room(seed=30 + q, room=r, steps=27, K=k) for q, (r, k) in enumerate([((26, 22, 18), 2), ((30, 20, 16), 4), ((20, 24, 41), 1)])]
ms = [run_gpu(c, "fp32", run=False) for c in cfgs]
with Group(ms) as grp:
    grp.set_branches(2)
    grp.run(27)
    out["group"] = [s.ir().tolist() for s in ms]
for s in ms:
    s.close()
print(json.dumps(out))
'''


def test_checked_library_exports_the_same_symbols():
    if not os.path.exists(CHECKED):
        pytest.skip("libfz_checked.so not built")
    from fases_b200 import _abi
    L = ctypes.CDLL(CHECKED)
    missing = [n for n in _abi.SIGNATURES if not hasattr(L, n)]
    assert not missing, missing


def _run(checked):
    env = dict(os.environ)
    env["FZ_BOUNDS_CHECK"] = "1" if checked else "0"
    r = subprocess.run([sys.executable, "-c", SCRIPT, ROOT], env=env, capture_output=True, text=True, timeout=600,
                       cwd=ROOT)
    assert r.returncode == 0, r.stderr[-3000:]
    return json.loads(r.stdout.strip().splitlines()[-1])


@pytest.mark.gpu
def test_checked_build_runs_clean_and_matches():
    if not os.path.exists(CHECKED):
        pytest.skip("libfz_checked.so not built")
    a = _run(True)
    b = _run(False)
    assert a.keys() == b.keys()
    for bands in (a.pop("bands"), b.pop("bands")):
        assert len(bands) == 6 and all(n == 3 for n in bands.values()), bands
    for k in a:
        if k.startswith("grad"):  # the adjoint's atomics sum in an order that varies from run to run
            for x, y in zip(a[k], b[k]):
                x, y = np.asarray(x), np.asarray(y)
                assert np.linalg.norm(x - y) <= 1e-5 * np.linalg.norm(y), k
        else:
            assert np.array_equal(np.asarray(a[k]), np.asarray(b[k])), k
