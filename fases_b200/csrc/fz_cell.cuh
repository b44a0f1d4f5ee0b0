// fz_cell.cuh -- per-cell parts of a stage shared by the stepping kernels: point sources, the cPML
// correction, the immersed ADE band. Products are contracted explicitly (fma), so that every kernel
// that runs these parts gives the same bits.
#pragma once
#include <cuda_runtime.h>
#include <math.h>

#include "fz_device.cuh"
#include "fz_pair.cuh"

namespace fz {

// Sum of the point sources of cell g at this stage (main3D.cu:1288, 1296, 1304).
template <class R>
__device__ __forceinline__ R source_sum(const StageArgs<R>& A, int64_t g) {
  const int64_t n = *A.step;
  const int64_t nn = A.nn_mul * n + A.nn_add;
  R add = R(0);
  for (int s = 0; s < A.nsrc; ++s) {
    if (A.src_cell[s] != g) continue;
    R amp;
    if (A.src_opt == 2) {
      const double ph = 2.0 * 3.14159265358979323846 * (double)A.src_freq[s] * (double)nn * (double)A.half_dt;
      amp = (R)sin(ph);
    } else {
      amp = (nn < A.n_us) ? A.u_s[nn] : R(0);
    }
    add += A.src_w * A.src_coef[s] * amp;
  }
  return add;
}

// cPML (functions3D.cuh:725-755): field += w dt ((1/kappa - 1) D + psi), psi frozen within the step
// and advanced once, in stage 2, by recursive convolution. D*: (X - Y, X + Y) of the
// characteristics' differences along each axis; cx, cy, cz: the cell's coefficients.
template <class R, int STAGE>
__device__ __forceinline__ void pml_axis(const StageArgs<R>& A, typename Pair<R>::T* psi, int64_t at,
                                         const PmlCoef<R>& c, typename Pair<R>::T D, R& p, R& vel) {
  const typename Pair<R>::T ps = psi[at];
  const R Dp = D.x * A.ih_p, Dv = D.y * A.ih_v;
  p = fma(A.wdt, fma(c.kinv1, Dp, ps.x), p);
  vel = fma(A.wdt, fma(c.kinv1, Dv, ps.y), vel);
  if (STAGE == 2) psi[at] = pmk(fma(c.b, ps.x, c.ca * Dp), fma(c.b, ps.y, c.ca * Dv));
}
template <class R, int STAGE>
__device__ __forceinline__ void pml_update(const StageArgs<R>& A, int i, int j, int k, const PmlCoef<R>& cx,
                                           const PmlCoef<R>& cy, const PmlCoef<R>& cz, typename Pair<R>::T Dx,
                                           typename Pair<R>::T Dy, typename Pair<R>::T Dz, R& p, R& u, R& v, R& w) {
  const int64_t d2 = A.pml_d2;
  if (cx.tile >= 0) {
    const int64_t X = cx.tile + d2 * ((int64_t)j + (int64_t)A.Ny * k);
    if (fz_inb(A.err, X, A.npsi[0])) pml_axis<R, STAGE>(A, A.psix, X, cx, Dx, p, u);
  }
  if (cy.tile >= 0) {
    const int64_t Y = (int64_t)i + (int64_t)A.Nx * ((int64_t)cy.tile + d2 * k);
    if (fz_inb(A.err, Y, A.npsi[1])) pml_axis<R, STAGE>(A, A.psiy, Y, cy, Dy, p, v);
  }
  if (cz.tile >= 0) {
    const int64_t Z = (int64_t)i + (int64_t)A.Nx * ((int64_t)j + (int64_t)A.Ny * cz.tile);
    if (fz_inb(A.err, Z, A.npsi[2])) pml_axis<R, STAGE>(A, A.psiz, Z, cz, Dz, p, w);
  }
}

// ------------------------------------------------------------------------------------------
// Immersed ADE band (functions3D.cuh:462-565 + ADE_solver 426-459), one thread per band cell of
// the compact list (or the thread that has just updated the cell). Probe geometry (normal, trilinear corner and weights at C - 2h n, chi) is
// precomputed once on the host. The probe reads the stage-input fields, which no kernel of this
// stage writes; the blend reads and writes only the band cell itself.
// ------------------------------------------------------------------------------------------
template <class R>
__device__ __forceinline__ R trilin(const R* __restrict__ f, int64_t q, int64_t Sx, int64_t plane, R sx,
                                    R sy, R sz) {
  const R ox = R(1) - sx, oy = R(1) - sy, oz = R(1) - sz;
  const R c00 = fma(__ldg(f + q + 1), sx, __ldg(f + q) * ox);
  const R c10 = fma(__ldg(f + q + Sx + 1), sx, __ldg(f + q + Sx) * ox);
  const R c01 = fma(__ldg(f + q + plane + 1), sx, __ldg(f + q + plane) * ox);
  const R c11 = fma(__ldg(f + q + plane + Sx + 1), sx, __ldg(f + q + plane + Sx) * ox);
  const R c0 = fma(c10, sy, c00 * oy), c1 = fma(c11, sy, c01 * oy);
  return fma(c1, sz, c0 * oz);
}

template <class R>
struct Vec4;
template <>
struct Vec4<float> {
  typedef float4 T;
};
template <>
struct Vec4<double> {
  typedef double4 T;
};

template <class R>
__device__ __forceinline__ bool band_inb(const BandArgs<R>& B, int64_t cell, const int4& rc) {
  return fz_inb(B.err, cell, B.nfield) && fz_inb(B.err, cell + rc.z, B.nfield) &&
         fz_inb(B.err, cell + rc.z + B.plane + B.Sx + 1, B.nfield);
}

// STAGE selects the ADE stage coefficients (a, b, c) = (0,1,1), (3,1,4), (1,2,3)
// (main3D.cu:1290, 1298, 1306): left = (a middle + b (right + dt L(right))) / c.
// KM, LM > 0: at most KM real poles and LM complex pairs. Every load that does not depend on the
// probe (the ADE states of the stage) is then issued at the top, beside the probe gathers, so one
// thread keeps ~50 loads in flight; KM = LM = 0 is the general form with the state loads inside the
// pole loops. (p, u, v, w): the cell's stage output on entry, the blended values on return.
template <class R, int STAGE, int KM, int LM>
__device__ __forceinline__ void band_cell(const BandArgs<R>& B, const int64_t b, const int64_t cell, const int4& rc,
                                          R& p, R& u, R& v, R& w) {
  typedef typename Vec4<R>::T V4;
  const int64_t q = cell + rc.z;
  const int m = rc.w;
  const int64_t nB = B.nB;
  const V4 g4 = reinterpret_cast<const V4*>(B.geo)[b];
  const V4 n4 = reinterpret_cast<const V4*>(B.nrm)[b];
  double rK[KM > 0 ? KM : 1], mK[KM > 0 ? KM : 1], r1L[LM > 0 ? LM : 1], r2L[LM > 0 ? LM : 1];
  double m1L[LM > 0 ? LM : 1], m2L[LM > 0 ? LM : 1];
#pragma unroll
  for (int k = 0; k < KM; ++k)
    if (k < B.K) {
      rK[k] = __ldg(B.phR + (int64_t)k * nB + b);
      if (STAGE > 0) mK[k] = __ldg(B.phM + (int64_t)k * nB + b);
    }
#pragma unroll
  for (int l = 0; l < LM; ++l)
    if (l < B.L) {
      r1L[l] = __ldg(B.s1R + (int64_t)l * nB + b);
      r2L[l] = __ldg(B.s2R + (int64_t)l * nB + b);
      if (STAGE > 0) {
        m1L[l] = __ldg(B.s1M + (int64_t)l * nB + b);
        m2L[l] = __ldg(B.s2M + (int64_t)l * nB + b);
      }
    }
  const R sx = g4.x, sy = g4.y, sz = g4.z, chi = g4.w;
  const R nx = n4.x, ny = n4.y, nz = n4.z;
  const R pD = trilin<R>(B.pi, q, B.Sx, B.plane, sx, sy, sz);
  const R uD = trilin<R>(B.ui, q, B.Sx, B.plane, sx, sy, sz);
  const R vD = trilin<R>(B.vi, q, B.Sx, B.plane, sx, sy, sz);
  const R wD = trilin<R>(B.wi, q, B.Sx, B.plane, sx, sy, sz);
  const R un = fma(wD, nz, fma(vD, ny, uD * nx));
  const R utx = fma(-un, nx, uD), uty = fma(-un, ny, vD), utz = fma(-un, nz, wD);
  const double wout = fma(B.Z0, (double)un, (double)pD);  // outgoing characteristic
  constexpr double a_ssp = (STAGE == 0) ? 0.0 : (STAGE == 1) ? 3.0 : 1.0;
  constexpr double b_ssp = (STAGE == 2) ? 2.0 : 1.0;
  constexpr double inv_c = (STAGE == 0) ? 1.0 : (STAGE == 1) ? 0.25 : 1.0 / 3.0;
  const double dt = B.dt;
  // one pole state of the ADE stage recursion: (a mid + b (r + dt L)) / c
  auto advance = [&](double r, double rate, double mid) {
    double x = b_ssp * fma(dt, rate, r);
    if (STAGE > 0) x = fma(a_ssp, mid, x);
    return x * inv_c;
  };
  double sumA = 0.0, sumBC = 0.0;
  auto real_pole = [&](int k, double r, double mid) {
    const int mi = m * B.K + k;
    const double x = advance(r, fma(-__ldg(B.zeta + mi), r, wout), mid);
    B.phL[(int64_t)k * nB + b] = x;
    sumA = fma(__ldg(B.A + mi), x, sumA);
  };
  auto pole_pair = [&](int l, double r1, double r2, double m1, double m2) {
    const int mi = m * B.L + l;
    const double al = __ldg(B.alpha + mi), be = __ldg(B.beta + mi);
    const double n1 = advance(r1, wout - fma(al, r1, be * r2), m1);
    const double n2 = advance(r2, fma(be, r1, -(al * r2)), m2);
    const int64_t si = (int64_t)l * nB + b;
    B.s1L[si] = n1;
    B.s2L[si] = n2;
    sumBC = fma(__ldg(B.B + mi), n1, fma(__ldg(B.C + mi), n2, sumBC));
  };
  if constexpr (KM > 0) {
#pragma unroll
    for (int k = 0; k < KM; ++k)
      if (k < B.K) real_pole(k, rK[k], STAGE > 0 ? mK[k] : 0.0);
#pragma unroll
    for (int l = 0; l < LM; ++l)
      if (l < B.L) pole_pair(l, r1L[l], r2L[l], STAGE > 0 ? m1L[l] : 0.0, STAGE > 0 ? m2L[l] : 0.0);
  } else {
    for (int k = 0; k < B.K; ++k) {
      const int64_t si = (int64_t)k * nB + b;
      real_pole(k, B.phR[si], STAGE > 0 ? B.phM[si] : 0.0);
    }
    for (int l = 0; l < B.L; ++l) {
      const int64_t si = (int64_t)l * nB + b;
      pole_pair(l, B.s1R[si], B.s2R[si], STAGE > 0 ? B.s1M[si] : 0.0, STAGE > 0 ? B.s2M[si] : 0.0);
    }
  }
  const double win = fma(__ldg(B.Rinf + m), wout, sumA + sumBC);  // incoming characteristic
  const R pb = (R)(0.5 * (win + wout));
  const R unb = (R)((wout - win) / (2.0 * B.Z0));
  const R omc = R(1) - chi;
  u = fma(chi, fma(unb, nx, utx), omc * u);
  v = fma(chi, fma(unb, ny, uty), omc * v);
  w = fma(chi, fma(unb, nz, utz), omc * w);
  p = fma(chi, pb, omc * p);
}

}  // namespace fz
