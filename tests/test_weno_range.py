"""The WENO centres over the range of their types. Smoothness indicators lie between eps and the square of
the largest difference, and the weights are formed from products of them: a very small eps (the 2D
legacy scheme takes any positive one) or very large fields must not carry those products out of the
type's range. Against the CPU oracle, which divides; FP64 to 1e-10 and FP32 to 1e-5, the tolerances of
the ordinary parity tests (a relative perturbation of 1e-15 of the start moves these FP64 runs by less
than 4e-15, and FP32 rounding in the oracle itself the FP32 ones by less than 9e-7)."""
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
