"""The WENO centres over the range of their types. Smoothness indicators lie between eps and the square of
the largest difference, and the weights are formed from products of them: a very small eps (the 2D
legacy scheme takes any positive one) or very large fields must not carry those products out of the
type's range. Against the CPU oracle, which divides; FP64 to 1e-10 and FP32 to 1e-5, the tolerances of
the ordinary parity tests (a relative perturbation of 1e-15 of the start moves these FP64 runs by less
than 4e-15, and FP32 rounding in the oracle itself the FP32 ones by less than 9e-7)."""
import ctypes
import json
import os
import subprocess
import sys

import numpy as np
import pytest

from tests.helpers import rel_l2, run_gpu, run_oracle, small_room
from tests.test_adjoint import STEPS, _cfg, _solver
from tests.test_legacy2d import _gpu, _oracle, _synthetic


@pytest.mark.gpu
@pytest.mark.parametrize("precision,eps,scale", [
    ("fp64", 1e-40, 1.0), ("fp64", 2e-39, 1.0), ("fp64", 1e-150, 1.0), ("fp64", 1e-7, 1e30), ("fp64", 1e-7, 1e70),
    ("fp64", 1e40, 1e25), ("fp32", 1e-19, 1.0), ("fp32", 6e-20, 1.0), ("fp32", 1e-7, 1e9)])
def test_legacy_scheme_at_the_ends_of_its_range(precision, eps, scale):
    fx = _synthetic(2)
    fx["eps"] = eps
    for k in ("p0", "u0", "v0"):
        fx[k] = fx[k] * scale
    ir_o, f_o = _oracle(fx, fx["Nt"])
    s = _gpu(fx, precision, fx["Nt"])
    tol = 1e-10 if precision == "fp64" else 1e-5
    got = [s.ir()] + list(s.fields())
    s.close()
    for a, b in zip(got, [ir_o] + list(f_o)):
        assert np.isfinite(a).all()
        assert rel_l2(a / scale, b / scale) < tol


@pytest.mark.gpu
@pytest.mark.parametrize("depth", [0, 5])  # the direct and the marching kernel
@pytest.mark.parametrize("scale", [1e20, 1e30, 1e70, 1e140])
def test_fp64_stepper_with_large_fields(scale, depth):
    cfg = small_room(seed=2, steps=60)
    cfg["p0"] = cfg["p0"] * scale
    cfg["sval"] = cfg["sval"] * scale
    o = run_oracle(cfg)
    s = run_gpu(cfg, "fp64", run=False)
    if depth:
        s.set_kz_chunk(depth)
    s.run(cfg["steps"])
    got = [s.ir()] + list(s.fields())
    s.close()
    for a, b in zip(got, [o.ir()[0]] + list(o.fields())):
        assert np.isfinite(a).all()
        assert rel_l2(a / scale, b / scale) < 1e-10


@pytest.mark.gpu
def test_fp64_gradient_scales_with_the_fields():
    """Where eps does not count, the traces are homogeneous of degree one in the fields and J and its
    gradient of degree two: with powers of two the same numbers but for the order of the sums (the probe
    scatter's atomics) and the cells below 1e-29 of the largest difference."""
    def gradient(scale):
        cfg = _cfg()
        cfg["p0"] = cfg["p0"] * scale
        cfg["sval"] = cfg["sval"] * scale
        s = _solver(cfg, "fp64")
        target = scale * 1e-3 * np.random.default_rng(8).standard_normal((len(cfg["recs"]), STEPS))
        g = s.misfit_gradient(target, segment_steps=16)
        s.close()
        return g

    a, b = 2.0 ** 76, 2.0 ** 183  # 7.6e22 and 1.2e55
    ga, gb = gradient(a), gradient(b)
    assert abs(gb["J"] / b ** 2 / (ga["J"] / a ** 2) - 1.0) < 1e-12
    for key in ("Rinf", "A", "zeta", "B", "C", "alpha", "beta"):
        x, y = np.asarray(ga[key]) / a ** 2, np.asarray(gb[key]) / b ** 2
        assert np.isfinite(y).all() and np.abs(x).max() > 0
        assert rel_l2(y, x) < 1e-10, key


HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
WAIT_TEST = os.path.join(ROOT, "fases_b200", "libfz_waittest.so")

RCP = r'''
import ctypes, json, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
from fases_b200 import _abi
L = _abi.lib()
L.fz_test_rcp.argtypes = [ctypes.POINTER(ctypes.c_double)] * 2 + [ctypes.c_int64]
L.fz_test_rcp.restype = ctypes.c_int
rng = np.random.default_rng(1)
m = np.concatenate([1.0 + rng.random(200000), [1.0, np.nextafter(1.0, 2.0), np.nextafter(2.0, 1.0), 1.5]])
out = {}
for name, lo, hi in (("indicators", -205, 340), ("range", -1020, 1020)):
    x = np.ldexp(m, rng.integers(lo, hi + 1, m.size))
    x = np.concatenate([x, [2.0 ** lo, 2.0 ** hi]])
    y = np.empty_like(x)
    p = lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))
    assert L.fz_test_rcp(p(x), p(y), x.size) == 0
    want = 1.0 / x
    out[name] = float((np.abs(y - want) / np.spacing(want)).max())
print(json.dumps(out))
'''


@pytest.mark.gpu
def test_fp64_reciprocal_against_division():
    """drcp over the products the centres give it and over all it takes: within one unit in the last place
    of the correctly rounded quotient (a seed of at least 20 bits and a third-order step leave 2^-60, the
    last operation's rounding half a unit, and the quotient's own rounding another half)."""
    if not os.path.exists(WAIT_TEST):
        pytest.skip("libfz_waittest.so not built")
    env = dict(os.environ, FZ_WAIT_TEST="1")
    env.pop("FZ_BOUNDS_CHECK", None)
    r = subprocess.run([sys.executable, "-c", RCP, ROOT], env=env, capture_output=True, text=True, timeout=300, cwd=ROOT)
    assert r.returncode == 0, r.stderr[-3000:]
    out = json.loads(r.stdout.strip().splitlines()[-1])
    assert all(v <= 1.0 for v in out.values()), out


def test_only_the_test_build_has_the_reciprocal_hook():
    if not os.path.exists(WAIT_TEST):
        pytest.skip("libfz_waittest.so not built")
    from fases_b200 import _abi
    assert hasattr(ctypes.CDLL(WAIT_TEST), "fz_test_rcp")
    assert not hasattr(ctypes.CDLL(_abi.LIB_PATH), "fz_test_rcp")
