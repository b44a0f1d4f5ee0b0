// fz_pair.cuh -- pair arithmetic shared by the stepping and adjoint kernels.
#pragma once
#include <cuda_runtime.h>
#include <math.h>

#include "fz_device.cuh"

namespace fz {

// ------------------------------------------------------------------------------------------
// Pair arithmetic. A pair holds the same quantity for two variables (pressure and the velocity
// component normal to the sweep), so every WENO-Z and flux operation runs on both at once. In
// FP32 these are the sm_100 paired instructions (add/mul/fma .f32x2).
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ float2 pmk(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ double2 pmk(double a, double b) { return make_double2(a, b); }
__device__ __forceinline__ float2 padd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 pmul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 pfma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 psub(float2 a, float2 b) {
  unsigned long long r;
  asm("sub.rn.f32x2 %0, %1, %2;"
      : "=l"(r)
      : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)));
  return *reinterpret_cast<float2*>(&r);
}
__device__ __forceinline__ float2 pabs(float2 a) { return make_float2(fabsf(a.x), fabsf(a.y)); }
__device__ __forceinline__ float frcp(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float2 prcp(float2 a) { return make_float2(frcp(a.x), frcp(a.y)); }
__device__ __forceinline__ float2 pswap(float2 a) { return make_float2(a.y, a.x); }

__device__ __forceinline__ double2 padd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 pmul(double2 a, double2 b) { return make_double2(a.x * b.x, a.y * b.y); }
__device__ __forceinline__ double2 pfma(double2 a, double2 b, double2 c) {
  return make_double2(fma(a.x, b.x, c.x), fma(a.y, b.y, c.y));
}
__device__ __forceinline__ double2 psub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 pabs(double2 a) { return make_double2(fabs(a.x), fabs(a.y)); }
__device__ __forceinline__ double2 pswap(double2 a) { return make_double2(a.y, a.x); }

template <class R>
__device__ __forceinline__ typename Pair<R>::T psplat(R x) {
  return pmk(x, x);
}

// ------------------------------------------------------------------------------------------
// WENO reconstruction at one cell centre: WENO-Z (Borges, Carmona, Costa & Don 2008, q = 1), the scheme
// of functions3D.cuh:763-1001 with the tables of main3D.cu:834-843 and eps = 1e-10 (main3D.cu:770).
//
// The reference evaluates V-(i+1/2) (idx = 1) and V+(i-1/2) (idx = 0) of a cell in two separate
// calls; both use the same three smoothness indicators and the same factors (1 + tau/(beta+eps)),
// and differ only in the linear weights d (mirrored) and the candidate rows. Both forms below evaluate
// them together, on the first differences a..d of the five-point stencil.
// ------------------------------------------------------------------------------------------
// FACES selects the face values computed: WENO_BOTH, or only V- (WENO_LO) or V+ (WENO_HI) where a
// caller uses one of them (the tile's halo rows); the value computed is the same either way.
constexpr int WENO_LO = 1, WENO_HI = 2, WENO_BOTH = 3;

// FP32, 3D solver: indicators from second differences D_r and one-sided first derivatives E_r,
//   candidates:  u_i + delta_r,   V = u_i + sum_r w_r delta_r,   w_r = d_r q_r / sum d q
//   12/13 beta_r = D_r^2 + 3/13 E_r^2
// (the 12/13 scaling is absorbed into eps). 45 paired operations; the form below takes 37 and the
// characteristics halve the exchange, 7 % of a large room's step, but another rounding than results
// this library has given before: traces and fields keep their bits.
template <int FACES = WENO_BOTH>
__device__ __forceinline__ void weno_center(float2 qm2, float2 qm1, float2 q0, float2 qp1, float2 qp2, float2& vm,
                                            float2& vp) {
  auto K = [](double x) { return make_float2((float)x, (float)x); };
  const float2 a = psub(qm1, qm2), b = psub(q0, qm1), c = psub(qp1, q0), d = psub(qp2, qp1);
  const float2 D2 = psub(b, a), D1 = psub(c, b), D0 = psub(d, c);
  const float2 E2 = pfma(b, K(2.0), D2);   // u_{i-2} - 4u_{i-1} + 3u_i
  const float2 E1 = padd(b, c);            // -(u_{i-1} - u_{i+1})
  const float2 E0 = pfma(c, K(-2.0), D0);  // 3u_i - 4u_{i+1} + u_{i+2} (sign)
  const float2 k313 = K(3.0 / 13.0), eps = K(1e-10 * 12.0 / 13.0), one = K(1.0);
  const float2 B0 = pfma(D0, D0, pfma(pmul(E0, k313), E0, eps));
  const float2 B1 = pfma(D1, D1, pfma(pmul(E1, k313), E1, eps));
  const float2 B2 = pfma(D2, D2, pfma(pmul(E2, k313), E2, eps));
  const float2 tau = pabs(psub(B0, B2));
  const float2 w0 = pfma(tau, prcp(B0), one);
  const float2 w1 = pfma(tau, prcp(B1), one);
  const float2 w2 = pfma(tau, prcp(B2), one);
  // normalisers: V- uses d = (3/10, 3/5, 1/10), V+ the mirrored (1/10, 3/5, 3/10); d_r delta_r for
  // both faces, written on the first and second differences
  const float2 t1 = pmul(w1, K(0.6)), h1 = pmul(D1, K(0.05));
  if constexpr ((FACES & WENO_LO) != 0) {
    const float2 S = pfma(w0, K(0.3), pfma(w2, K(0.1), t1));
    const float2 e0 = pfma(c, K(0.15), pmul(D0, K(-0.05)));
    const float2 e1 = pfma(E1, K(0.15), h1);
    const float2 e2 = pfma(b, K(0.05), pmul(D2, K(1.0 / 30.0)));
    vm = pfma(pfma(w2, e2, pfma(w1, e1, pmul(w0, e0))), prcp(S), q0);
  }
  if constexpr ((FACES & WENO_HI) != 0) {
    const float2 S = pfma(w0, K(0.1), pfma(w2, K(0.3), t1));
    const float2 e0 = pfma(c, K(-0.05), pmul(D0, K(1.0 / 30.0)));
    const float2 e1 = pfma(E1, K(-0.15), h1);
    const float2 e2 = pfma(b, K(-0.15), pmul(D2, K(-0.05)));
    vp = pfma(pfma(w2, e2, pfma(w1, e1, pmul(w0, e0))), prcp(S), q0);
  }
}

// FP64, and the 2D legacy scheme: multiplied out, the indicators are quadratic forms of neighbouring
// differences,
//   3/4 beta_2 = a^2 - 11/4 a b + 5/2 b^2    3/4 beta_1 = b^2 - 5/4 b c + c^2
//   3/4 beta_0 = 5/2 c^2 - 11/4 c d + d^2
// (beta_1 is at least 0.6 of its larger square, the others at least 0.24 d^2 or a^2 and 0.6 c^2 or b^2, so
// rounding cannot make one negative; the 3/4 goes into eps), and the weighted candidates 5 d_r (V_r - u_i), scaled so that most coefficients are 1:
//   V-: c - d/4, c + b/2, (5 b - 2 a)/12      V+: -(5 c - 2 d)/12, -(b + c/2), -(b - a/4)
// with the normaliser 5 sum d_r q_r: 37 operations a centre for both faces.
// Nonlinear weights from the indicators B_r = 3/4 (beta_r + eps), up to a factor common to the three
// (it cancels between the sums and their normalisers).
//
// Products of indicators leave the range of the type long before the indicators do (B lies between eps
// and the square of the largest difference), so each form scales by a power of two, which is exact (but
// for what falls below the smallest normal number): a 2D solve with eps = 1e-40, or fields of 1e30, are as
// good as any.

// 2^-e for x = m 2^e, m in [1, 2), given x's upper word (FP64) or bits (FP32); x subnormal or zero: the
// largest power of two (FP32: x finite)
__device__ __forceinline__ double pow2_inverse64(int hi) {
  return __hiloint2double(max((2046 << 20) - (hi & 0x7ff00000), 1 << 20), 0);
}
__device__ __forceinline__ float pow2_inverse32(int bits) {
  return __int_as_float((254 << 23) - (bits & 0x7f800000));
}

// Reciprocal in 64 bits: the hardware's coarse seed (at least 20 bits) and one third-order
// Householder step r (1 + e + e^2), e = 1 - x r, which leaves an error of e^3 < 2^-59 beside the
// rounding of the last operation. For normal x below 2^1022 (no scaling, no special cases).
__device__ __forceinline__ double drcp(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double e = fma(-x, r, 1.0);
  return fma(r, fma(e, e, e), r);
}

struct WenoZ {  // 1 + tau / B_r, tau = |B_0 - B_2|
  // In FP64 a reciprocal costs several FMA-pipe operations: the factors times B_0 B_1 B_2. The weighted
  // sums go up to B^3.5, so indicators from 2^256 on, differences above 1e38, are taken over the largest
  // one's power of two, with a floor of 2^-256 (differences 1e-38 of the largest) in the place of the
  // scaled eps. B_1 is at most 2.7 times the sum of the others. One test for both variables of a centre
  // (190 x 150 x 140 cells: 1.5 % of a step; a test for each, which keeps their chains from being
  // interleaved, 5 %; the products scaled without a test, 1.9 % and good to 1e94 only).
  static constexpr int WIDE = (1023 + 256) << 20;
  static __device__ __forceinline__ void range(double2& B0, double2& B1, double2& B2) {
    const int x = max(__double2hiint(B0.x), __double2hiint(B2.x)), y = max(__double2hiint(B0.y), __double2hiint(B2.y));
    if (max(x, y) >= WIDE) {
      const double2 s = make_double2(pow2_inverse64(x), pow2_inverse64(y));
      const double f = __hiloint2double((1023 - 256) << 20, 0);
      B0 = pfma(B0, s, make_double2(f, f));
      B1 = pfma(B1, s, make_double2(f, f));
      B2 = pfma(B2, s, make_double2(f, f));
    }
  }
  __device__ __forceinline__ void operator()(double B0, double B1, double B2, double& w0, double& w1, double& w2) const {
    const double tau = fabs(B0 - B2);
    const double B12 = B1 * B2, B02 = B0 * B2, B01 = B0 * B1, B012 = B0 * B12;
    w0 = fma(tau, B12, B012);
    w1 = fma(tau, B02, B012);
    w2 = fma(tau, B01, B012);
  }
};
// 1 / B_r^2 (Jiang & Shu 1996), over the power of two of the largest (803 x 815 nodes FP32: 1.2 of 52.7 us a
// step)
struct WenoJS {
  static __device__ __forceinline__ void scaled(float r0, float r1, float r2, float& w0, float& w1, float& w2) {
    const float s = pow2_inverse32(max(max(__float_as_int(r0), __float_as_int(r1)), __float_as_int(r2)));
    w0 = r0 * s;
    w1 = r1 * s;
    w2 = r2 * s;
  }
  __device__ __forceinline__ void operator()(float2 B0, float2 B1, float2 B2, float2& w0, float2& w1, float2& w2) const {
    const float2 r0 = prcp(B0), r1 = prcp(B1), r2 = prcp(B2);
    float2 q0, q1, q2;
    scaled(r0.x, r1.x, r2.x, q0.x, q1.x, q2.x);
    scaled(r0.y, r1.y, r2.y, q0.y, q1.y, q2.y);
    w0 = pmul(q0, q0);
    w1 = pmul(q1, q1);
    w2 = pmul(q2, q2);
  }
  static __device__ __forceinline__ void range(double2&, double2&, double2&) {}
  __device__ __forceinline__ void operator()(double B0, double B1, double B2, double& w0, double& w1, double& w2) const {
    const double P0 = B1 * B2, P1 = B0 * B2, P2 = B0 * B1;
    const double s = pow2_inverse64(max(max(__double2hiint(P0), __double2hiint(P1)), __double2hiint(P2)));
    const double q0 = P0 * s, q1 = P1 * s, q2 = P2 * s;
    w0 = q0 * q0;
    w1 = q1 * q1;
    w2 = q2 * q2;
  }
};

// The weighted sums and normalisers of a centre: V- = q0 + Nm / Sm, V+ = q0 - Np / Sp. eps: 3/4 of the
// scheme's.
template <int FACES, class W>
__device__ __forceinline__ void weno_sums(float2 qm2, float2 qm1, float2 q0, float2 qp1, float2 qp2, float eps,
                                          W weights, float2& Nm, float2& Np, float2& rSm, float2& rSp) {
  auto K = [](float x) { return make_float2(x, x); };
  const float2 a = psub(qm1, qm2), b = psub(q0, qm1), c = psub(qp1, q0), d = psub(qp2, qp1);
  const float2 bb = pfma(b, b, K(eps));
  const float2 B1 = pfma(c, pfma(b, K(-1.25f), c), bb);
  const float2 B2 = pfma(a, pfma(b, K(-2.75f), a), pfma(bb, K(2.5f), K(-1.5f * eps)));
  const float2 B0 = pfma(d, pfma(c, K(-2.75f), d), pfma(pmul(c, K(2.5f)), c, K(eps)));
  float2 w0, w1, w2;
  weights(B0, B1, B2, w0, w1, w2);
  const float2 t1 = pmul(w1, K(3.f));
  if constexpr ((FACES & WENO_LO) != 0) {
    rSm = prcp(pfma(w0, K(1.5f), pfma(w2, K(0.5f), t1)));
    const float2 e0 = pfma(d, K(-0.25f), c), e1 = pfma(b, K(0.5f), c);
    const float2 e2 = pfma(a, K((float)(-1.0 / 6.0)), pmul(b, K((float)(5.0 / 12.0))));
    Nm = pfma(w2, e2, pfma(w1, e1, pmul(w0, e0)));
  }
  if constexpr ((FACES & WENO_HI) != 0) {
    rSp = prcp(pfma(w0, K(0.5f), pfma(w2, K(1.5f), t1)));
    const float2 g0 = pfma(d, K((float)(-1.0 / 6.0)), pmul(c, K((float)(5.0 / 12.0))));
    const float2 g1 = pfma(c, K(0.5f), b), g2 = pfma(a, K(-0.25f), b);
    Np = pfma(w2, g2, pfma(w1, g1, pmul(w0, g0)));
  }
}

// In FP64 the weights come without reciprocals (above): 2 instead of 5 per variable (190 x 150 x 140 cells:
// a stage 0.175-0.183 ms instead of 0.265-0.272; both normalisers on one reciprocal take the same time).
template <int FACES, class W>
__device__ __forceinline__ void weno_sums1(double a, double b, double c, double d, double B0, double B1, double B2,
                                           W weights, double& Nm, double& Np, double& rSm, double& rSp) {
  double w0, w1, w2;
  weights(B0, B1, B2, w0, w1, w2);
  const double t1 = 3.0 * w1;
  if constexpr ((FACES & WENO_LO) != 0) {
    rSm = drcp(fma(w0, 1.5, fma(w2, 0.5, t1)));
    const double e0 = fma(d, -0.25, c), e1 = fma(b, 0.5, c), e2 = fma(a, -1.0 / 6.0, b * (5.0 / 12.0));
    Nm = fma(w2, e2, fma(w1, e1, w0 * e0));
  }
  if constexpr ((FACES & WENO_HI) != 0) {
    rSp = drcp(fma(w0, 0.5, fma(w2, 1.5, t1)));
    const double g0 = fma(d, -1.0 / 6.0, c * (5.0 / 12.0)), g1 = fma(c, 0.5, b), g2 = fma(a, -0.25, b);
    Np = fma(w2, g2, fma(w1, g1, w0 * g0));
  }
}
template <int FACES, class W>
__device__ __forceinline__ void weno_sums(double2 qm2, double2 qm1, double2 q0, double2 qp1, double2 qp2, double eps,
                                          W weights, double2& Nm, double2& Np, double2& rSm, double2& rSp) {
  auto K = [](double x) { return make_double2(x, x); };
  const double2 a = psub(qm1, qm2), b = psub(q0, qm1), c = psub(qp1, q0), d = psub(qp2, qp1);
  const double2 bb = pfma(b, b, K(eps));
  double2 B1 = pfma(c, pfma(b, K(-1.25), c), bb);
  double2 B2 = pfma(a, pfma(b, K(-2.75), a), pfma(bb, K(2.5), K(-1.5 * eps)));
  double2 B0 = pfma(d, pfma(c, K(-2.75), d), pfma(pmul(c, K(2.5)), c, K(eps)));
  W::range(B0, B1, B2);
  weno_sums1<FACES>(a.x, b.x, c.x, d.x, B0.x, B1.x, B2.x, weights, Nm.x, Np.x, rSm.x, rSp.x);
  weno_sums1<FACES>(a.y, b.y, c.y, d.y, B0.y, B1.y, B2.y, weights, Nm.y, Np.y, rSm.y, rSp.y);
}

// Outgoing characteristics of a centre, all the Godunov flux needs of it (functions3D.cuh:56-78 with
// p and Z0 q, Z0 = rho c): the right-going one at the face above, wr = p + Z0 q of V-(i+1/2), and the
// left-going one at the face below, wl = p - Z0 q of V+(i-1/2). The flux through a face is
//   F_p = c/2 (wr(i) - wl(i+1)),   F_q = 1/(2 rho) (wr(i) + wl(i+1)),
// so centres exchange two numbers instead of four.
template <class R, int FACES = WENO_BOTH, class W = WenoZ>
__device__ __forceinline__ void weno_waves(typename Pair<R>::T qm2, typename Pair<R>::T qm1, typename Pair<R>::T q0,
                                           typename Pair<R>::T qp1, typename Pair<R>::T qp2, R Z0, R& wr, R& wl,
                                           R eps = R(0.75e-10)) {
  typename Pair<R>::T Nm, Np, rm, rp;
  weno_sums<FACES>(qm2, qm1, q0, qp1, qp2, eps, W(), Nm, Np, rm, rp);
  if constexpr ((FACES & WENO_LO) != 0) wr = fma(Z0, fma(Nm.y, rm.y, q0.y), fma(Nm.x, rm.x, q0.x));
  if constexpr ((FACES & WENO_HI) != 0) wl = fma(-Z0, fma(-Np.y, rp.y, q0.y), fma(-Np.x, rp.x, q0.x));
}

__device__ __forceinline__ void weno_center(double2 qm2, double2 qm1, double2 q0, double2 qp1, double2 qp2, double2& vm,
                                            double2& vp) {
  double2 Nm, Np, rm, rp;
  weno_sums<WENO_BOTH>(qm2, qm1, q0, qp1, qp2, 0.75e-10, WenoZ(), Nm, Np, rm, rp);
  vm = pfma(Nm, rm, q0);
  vp = psub(q0, pmul(Np, rp));
}

// Godunov (exact Riemann) flux of linear acoustics for a (pressure, normal velocity) pair
// (functions3D.cuh:56-78):  F_p = 1/2 (rho c^2 (q+ + q-) - c (p+ - p-)),
//                           F_q = 1/2 ((p+ + p-)/rho - c (q+ - q-)).
template <class R>
__device__ __forceinline__ typename Pair<R>::T godunov(typename Pair<R>::T vm, typename Pair<R>::T vp,
                                                       typename Pair<R>::T kA, typename Pair<R>::T kC) {
  const typename Pair<R>::T sum = padd(vm, vp), dif = psub(vp, vm);
  return pfma(dif, kC, pmul(pswap(sum), kA));
}

// Difference of the Godunov fluxes through the low and the high face of a cell, F(lo) - F(hi),
// from the face states (left state of a face = V- of the centre below it, right state = V+ of the
// centre above): the flux is linear in the states, so the difference is taken on the sums and
// differences first and swapped and scaled once.
template <class R>
__device__ __forceinline__ typename Pair<R>::T godunov_diff(typename Pair<R>::T vm_lo, typename Pair<R>::T vp_lo,
                                                            typename Pair<R>::T vm_hi, typename Pair<R>::T vp_hi,
                                                            typename Pair<R>::T kA, typename Pair<R>::T kC) {
  const typename Pair<R>::T S = psub(padd(vm_lo, vp_lo), padd(vm_hi, vp_hi));
  const typename Pair<R>::T D = psub(psub(vp_lo, vm_lo), psub(vp_hi, vm_hi));
  return pfma(D, kC, pmul(pswap(S), kA));
}

// What the stage kernels pass between centres. A centre gives X lo for the face above it and X hi for
// the face below; face() joins the lo of a centre and the hi of the one above it; the differences across
// a cell (low minus high face) come as a (pressure, velocity) pair to be scaled by dt_p, dt_v.
template <class R>
struct Sweep;
// FP32: both face states, and the flux differences of the states.
template <>
struct Sweep<float> {
  typedef float2 X;
  typedef float2 F;  // a face's flux
  template <int FACES = WENO_BOTH, class A>
  static __device__ __forceinline__ void centre(const A&, float2 qm2, float2 qm1, float2 q0, float2 qp1, float2 qp2,
                                                X& lo, X& hi) {
    weno_center<FACES>(qm2, qm1, q0, qp1, qp2, lo, hi);
  }
  template <class A>
  static __device__ __forceinline__ F face(const A& a, X lo, X hi) {
    return godunov<float>(lo, hi, pmk(a.frc2, a.firho), psplat<float>(-a.fc));
  }
  static __device__ __forceinline__ float2 across(F below, F above) { return psub(below, above); }
  // from the states: lo of the centre below, own hi, own lo, hi of the centre above
  template <class A>
  static __device__ __forceinline__ float2 across(const A& a, X lo_below, X hi, X lo, X hi_above) {
    return godunov_diff<float>(lo_below, hi, lo, hi_above, pmk(a.frc2, a.firho), psplat<float>(-a.fc));
  }
};
// FP64: the characteristics wr, wl. (X - Y, X + Y) of their differences.
template <>
struct Sweep<double> {
  typedef double X;
  typedef double2 F;  // (wr of the centre below, wl of the centre above)
  template <int FACES = WENO_BOTH, class A>
  static __device__ __forceinline__ void centre(const A& a, double2 qm2, double2 qm1, double2 q0, double2 qp1,
                                                double2 qp2, X& lo, X& hi) {
    weno_waves<double, FACES>(qm2, qm1, q0, qp1, qp2, a.z0, lo, hi);
  }
  template <class A>
  static __device__ __forceinline__ F face(const A&, X lo, X hi) {
    return make_double2(lo, hi);
  }
  static __device__ __forceinline__ double2 across(F below, F above) {
    const double x = below.x - above.x, y = below.y - above.y;
    return make_double2(x - y, x + y);
  }
  template <class A>
  static __device__ __forceinline__ double2 across(const A&, X lo_below, X hi, X lo, X hi_above) {
    return across(make_double2(lo_below, hi), make_double2(lo, hi_above));
  }
};
__device__ __forceinline__ float shfl_up1(float x) { return __shfl_up_sync(0xffffffffu, x, 1); }
__device__ __forceinline__ float2 shfl_up1(float2 x) { return make_float2(shfl_up1(x.x), shfl_up1(x.y)); }
__device__ __forceinline__ double shfl_up1(double x) { return __shfl_up_sync(0xffffffffu, x, 1); }
__device__ __forceinline__ float shfl_down1(float x) { return __shfl_down_sync(0xffffffffu, x, 1); }
__device__ __forceinline__ float2 shfl_down1(float2 x) { return make_float2(shfl_down1(x.x), shfl_down1(x.y)); }
__device__ __forceinline__ double shfl_down1(double x) { return __shfl_down_sync(0xffffffffu, x, 1); }

}  // namespace fz
