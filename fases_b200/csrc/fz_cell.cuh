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

// Receiver samples of a completed step (main3D.cu:1399-1414) into trace column n, by the threads
// t = 0 .. nt-1; a non-finite sample sets the health word.
template <class R>
__device__ __forceinline__ void record_samples(const R* p, const R* u, const R* v, const R* w, const int64_t* rcell,
                                               int nrec, double* ir, double* vel, int64_t cap, int64_t n,
                                               int32_t* err, int64_t nfield, int t, int nt) {
  for (int r = t; r < nrec; r += nt) {
    const int64_t c = rcell[r];
    if (!fz_inb(err, c, nfield)) continue;
    const double pp = (double)p[c], uu = (double)u[c], vv = (double)v[c], ww = (double)w[c];
    // health word: a blown-up solution reaches the receivers (their samples are read anyway)
    if (!isfinite(pp) || !isfinite(uu) || !isfinite(vv) || !isfinite(ww)) atomicOr(err, KERR_NONFINITE);
    if (n < cap) {
      const int64_t o = (int64_t)r * cap + n;
      ir[o] = pp;
      vel[3 * o + 0] = uu;
      vel[3 * o + 1] = vv;
      vel[3 * o + 2] = ww;
    }
  }
}
// The previous step's samples, by the threads of one block of a stage 0 launch: the step's result is
// the stage's input, so this needs no launch of its own between the steps. Many receivers lengthen that
// block, about as much as they did their own launch: us a step with 16 / 4096 / 20000 receivers, by a launch
// -> here, 26 x 22 x 18 FP32 74 / 94 / 171 -> 15 / 38 / 125, 119 x 103 x 87 130 / 155 / 253 -> 122 / 144 / 251,
// 250 x 200 x 150 582 / 608 / 713 -> 556 / 559 / 651, where other blocks hide part of it.
template <class R>
__device__ __noinline__ void stage_receivers(const StageArgs<R>& A, int t, int nt) {
  record_samples<R>(A.pi, A.ui, A.vi, A.wi, A.rcell, A.rec_n, A.ir, A.vel, A.rec_cap, *A.step + A.rec_off, A.err,
                    A.nfield, t, nt);
}

// cPML (functions3D.cuh:725-755): field += w dt ((1/kappa - 1) D + psi), psi frozen within the step
// and advanced once, in stage 2, by recursive convolution. D*: the differences
// along each axis as Sweep gives them; cx, cy, cz: the cell's coefficients.
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
  const R c00 = fma(__ldg(f + q), ox, __ldg(f + q + 1) * sx);
  const R c10 = fma(__ldg(f + q + Sx), ox, __ldg(f + q + Sx + 1) * sx);
  const R c01 = fma(__ldg(f + q + plane), ox, __ldg(f + q + plane + 1) * sx);
  const R c11 = fma(__ldg(f + q + plane + Sx), ox, __ldg(f + q + plane + Sx + 1) * sx);
  const R c0 = fma(c00, oy, c10 * sy), c1 = fma(c01, oy, c11 * sy);
  return fma(c0, oz, c1 * sz);
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

// One pole state of an ADE stage, left = (a middle + b (right + dt L(right))) / c with the stage's
// (a, b, c) = (0,1,1), (3,1,4), (1,2,3) (main3D.cu:1290, 1298, 1306), given the rate L(right).
template <int STAGE>
__device__ __forceinline__ double ade_advance(double right, double rate, double mid, double dt) {
  constexpr double a = (STAGE == 0) ? 0.0 : (STAGE == 1) ? 3.0 : 1.0;
  constexpr double b = (STAGE == 2) ? 2.0 : 1.0;
  constexpr double inv_c = (STAGE == 0) ? 1.0 : (STAGE == 1) ? 0.25 : 1.0 / 3.0;
  double x = b * fma(dt, rate, right);
  if (STAGE > 0) x = fma(a, mid, x);
  return x * inv_c;
}
template <int STAGE>
__device__ __forceinline__ double ade_real(double right, double mid, double zeta, double wout, double dt) {
  return ade_advance<STAGE>(right, fma(-zeta, right, wout), mid, dt);
}
template <int STAGE>
__device__ __forceinline__ void ade_pair(double& r1, double& r2, double m1, double m2, double al, double be,
                                         double wout, double dt) {
  const double n1 = ade_advance<STAGE>(r1, wout - fma(al, r1, be * r2), m1, dt);
  r2 = ade_advance<STAGE>(r2, fma(be, r1, -(al * r2)), m2, dt);
  r1 = n1;
}

// The band cell b at `cell`: (p, u, v, w) is the cell's stage output on entry, the blended values on
// return.
// KEEP: the pole states after this stage are stored (the left role), and the stage reads its right and
// middle sets. Otherwise only the last stage stores states: the recursion is linear in the state at
// step start and the outgoing characteristics, so stages 1 and 2 recompute the earlier stages' states
// from those (8 bytes a stage, kept in wst) instead of reading and writing sets of 8 (K + 2L) bytes: every
// stage reads the set of step start. With K = L = 2 a band cell moves 232 instead of 384 bytes of states
// and characteristics a step, with the same bits:
// 500 x 400 x 200 cells (2.35 M band cells) 120 us a launch instead of 137, 190 x 150 x 140 FP64 39
// instead of 44. By its counters (192^3) the kernel then reads 230 to 246 bytes of DRAM a cell and launch,
// 55 to 59 % of the peak rate: band rows of walls normal to x are three cells long, a third of a sector.
// KM, LM > 0: at most KM real poles and LM complex pairs. Every load that does not depend on the
// probe is then issued at the top, beside the probe gathers, so one thread keeps ~50 loads in flight;
// KM = LM = 0 is the general form with the state loads inside the pole loops; it keeps every state.
template <class R, int STAGE, int KM, int LM, bool KEEP>
__device__ __forceinline__ void band_cell(const BandArgs<R>& B, const int64_t b, const int64_t cell, const int4& rc,
                                          R& p, R& u, R& v, R& w) {
  typedef typename Vec4<R>::T V4;
  const int64_t q = cell + rc.z;
  const int m = rc.w;
  const int64_t nB = B.nB;
  const V4 g4 = reinterpret_cast<const V4*>(B.geo)[b];
  const V4 n4 = reinterpret_cast<const V4*>(B.nrm)[b];
  constexpr bool RIGHT = KEEP && STAGE > 0;  // the right set is not the step-start (middle) one
  double rK[KM > 0 ? KM : 1], mK[KM > 0 ? KM : 1], r1L[LM > 0 ? LM : 1], r2L[LM > 0 ? LM : 1];
  double m1L[LM > 0 ? LM : 1], m2L[LM > 0 ? LM : 1];
#pragma unroll
  for (int k = 0; k < KM; ++k)
    if (k < B.K) {
      mK[k] = __ldg(B.phM + (int64_t)k * nB + b);
      if (RIGHT) rK[k] = __ldg(B.phR + (int64_t)k * nB + b);
    }
#pragma unroll
  for (int l = 0; l < LM; ++l)
    if (l < B.L) {
      m1L[l] = __ldg(B.s1M + (int64_t)l * nB + b);
      m2L[l] = __ldg(B.s2M + (int64_t)l * nB + b);
      if (RIGHT) {
        r1L[l] = __ldg(B.s1R + (int64_t)l * nB + b);
        r2L[l] = __ldg(B.s2R + (int64_t)l * nB + b);
      }
    }
  double w0 = 0.0, w1 = 0.0;  // the outgoing characteristics of the earlier stages
  if (KM > 0 && !KEEP && STAGE > 0) w0 = __ldg(B.wst + b);
  if (KM > 0 && !KEEP && STAGE > 1) w1 = __ldg(B.wst + nB + b);
  const R sx = g4.x, sy = g4.y, sz = g4.z, chi = g4.w;
  const R nx = n4.x, ny = n4.y, nz = n4.z;
  const R pD = trilin<R>(B.pi, q, B.Sx, B.plane, sx, sy, sz);
  const R uD = trilin<R>(B.ui, q, B.Sx, B.plane, sx, sy, sz);
  const R vD = trilin<R>(B.vi, q, B.Sx, B.plane, sx, sy, sz);
  const R wD = trilin<R>(B.wi, q, B.Sx, B.plane, sx, sy, sz);
  const R un = fma(wD, nz, fma(uD, nx, vD * ny));
  const R utx = fma(-un, nx, uD), uty = fma(-un, ny, vD), utz = fma(-un, nz, wD);
  const double wout = fma(B.Z0, (double)un, (double)pD);  // outgoing characteristic
  if (KM > 0 && !KEEP && STAGE < 2) B.wst[STAGE * nB + b] = wout;
  const double dt = B.dt;
  double sumA = 0.0, sumBC = 0.0;
  auto real_pole = [&](int k, double r, double mid) {
    const int mi = m * B.K + k;
    const double zeta = __ldg(B.zeta + mi);
    if (!RIGHT) r = mid;
    if (!KEEP && STAGE > 0) r = ade_real<0>(r, mid, zeta, w0, dt);
    if (!KEEP && STAGE > 1) r = ade_real<1>(r, mid, zeta, w1, dt);
    r = ade_real<STAGE>(r, mid, zeta, wout, dt);
    if (KEEP || STAGE == 2) B.phL[(int64_t)k * nB + b] = r;
    sumA = fma(__ldg(B.A + mi), r, sumA);
  };
  auto pole_pair = [&](int l, double r1, double r2, double m1, double m2) {
    const int mi = m * B.L + l;
    const double al = __ldg(B.alpha + mi), be = __ldg(B.beta + mi);
    if (!RIGHT) {
      r1 = m1;
      r2 = m2;
    }
    if (!KEEP && STAGE > 0) ade_pair<0>(r1, r2, m1, m2, al, be, w0, dt);
    if (!KEEP && STAGE > 1) ade_pair<1>(r1, r2, m1, m2, al, be, w1, dt);
    ade_pair<STAGE>(r1, r2, m1, m2, al, be, wout, dt);
    const int64_t si = (int64_t)l * nB + b;
    if (KEEP || STAGE == 2) {
      B.s1L[si] = r1;
      B.s2L[si] = r2;
    }
    sumBC += fma(__ldg(B.B + mi), r1, __ldg(B.C + mi) * r2);
  };
  if constexpr (KM > 0) {
#pragma unroll
    for (int k = 0; k < KM; ++k)
      if (k < B.K) real_pole(k, rK[k], mK[k]);
#pragma unroll
    for (int l = 0; l < LM; ++l)
      if (l < B.L) pole_pair(l, r1L[l], r2L[l], m1L[l], m2L[l]);
  }
  double win;  // incoming characteristic
  if constexpr (KM > 0) {
    win = fma(__ldg(B.Rinf + m), wout, sumA) + sumBC;
  } else {
    // any number of poles: the states after every stage are kept, the products left to the compiler to
    // contract, as this form has always been built
    constexpr double a_ssp = (STAGE == 0) ? 0.0 : (STAGE == 1) ? 3.0 : 1.0;
    constexpr double b_ssp = (STAGE == 2) ? 2.0 : 1.0;
    constexpr double inv_c = (STAGE == 0) ? 1.0 : (STAGE == 1) ? 0.25 : 1.0 / 3.0;
    auto real = [&](int k, double r, double mid) {
      const int mi = m * B.K + k;
      const double Lphi = wout - __ldg(B.zeta + mi) * r;
      double v = b_ssp * (r + B.dt * Lphi);
      if (STAGE > 0) v += a_ssp * mid;
      v *= inv_c;
      B.phL[(int64_t)k * nB + b] = v;
      sumA += __ldg(B.A + mi) * v;
    };
    auto pair = [&](int l, double r1, double r2, double m1, double m2) {
      const int mi = m * B.L + l;
      const double al = __ldg(B.alpha + mi), be = __ldg(B.beta + mi);
      const double L1 = wout - (al * r1 + be * r2);
      const double L2 = be * r1 - al * r2;
      double n1 = b_ssp * (r1 + B.dt * L1);
      double n2 = b_ssp * (r2 + B.dt * L2);
      if (STAGE > 0) {
        n1 += a_ssp * m1;
        n2 += a_ssp * m2;
      }
      n1 *= inv_c;
      n2 *= inv_c;
      const int64_t si = (int64_t)l * nB + b;
      B.s1L[si] = n1;
      B.s2L[si] = n2;
      sumBC += __ldg(B.B + mi) * n1 + __ldg(B.C + mi) * n2;
    };
    for (int k = 0; k < B.K; ++k) {
      const int64_t si = (int64_t)k * nB + b;
      real(k, B.phR[si], STAGE > 0 ? B.phM[si] : 0.0);
    }
    for (int l = 0; l < B.L; ++l) {
      const int64_t si = (int64_t)l * nB + b;
      pair(l, B.s1R[si], B.s2R[si], STAGE > 0 ? B.s1M[si] : 0.0, STAGE > 0 ? B.s2M[si] : 0.0);
    }
    win = __ldg(B.Rinf + m) * wout + sumA + sumBC;
  }
  const R pb = (R)(0.5 * (win + wout));
  const R unb = (R)((wout - win) / (2.0 * B.Z0));
  const R omc = R(1) - chi;
  u = fma(omc, u, chi * fma(unb, nx, utx));
  v = fma(omc, v, chi * fma(unb, ny, uty));
  // (which product is the rounded one differs between the forms, as they have always been contracted)
  const R wb = fma(unb, nz, utz);
  w = KM > 0 ? fma(omc, w, chi * wb) : fma(chi, wb, omc * w);
  p = fma(omc, p, chi * pb);
}

}  // namespace fz
