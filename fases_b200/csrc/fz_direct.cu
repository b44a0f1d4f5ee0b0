// fz_direct.cu -- the stage of a small room: one warp-autonomous kernel per stage for rooms that
// cannot fill the GPU with the marching tiles of fz_kernels.cu.
//
// The marching kernel (32 x 16 columns, one barrier a plane, TMA tiles) needs hundreds of CTAs of
// many planes to run well; a room of 10^4 to 10^6 cells gives it a handful of CTAs whose planes run
// one after another (26 x 22 x 18 cells: 4 CTAs x 9 planes, 25 us a stage; 71 x 53 x 47: 60 CTAs x 10
// planes, 28 us), and the band list one more dependent launch. Here
//  - a warp owns 30 cells of a row (lanes 0 and 31 are the halo centres): x centres once per lane,
//    exchanged by shuffles; y and z centres of the rows below and above recomputed (three a cell instead
//    of one). No shared memory, no barrier: all loads of a cell are independent and hit L1 / L2;
//  - the thread that updated a band cell runs its ADE boundary at once (the probe reads the stage
//    input), which saves the band launch.
// About twice the marching kernel's arithmetic a cell, so it is the better one only while the GPU is
// not full; use_direct (fz_api.cpp) draws the line. 26 x 22 x 18 FP32 takes 15 to 16 us a step (marching in
// chunks of 9 planes: 72), 45 x 38 x 29 FP64 26 (10 planes: 107). What is left is the latency of the
// chained loads (stencil, band record, probe: five to six of the ten cycles between two instructions of a
// warp, by its stall counters) and the launches. Five or six CTAs an SM (96, 80 registers) measured 17
// and 18 us; programmatic dependent launches 16.7 where plain ones took 16.0.
// A planar room marches along y, a warp one row or (FP64 planes near the line) two: no barrier there, and
// the second row's centres come from the first's registers.
#include <cuda_runtime.h>

#include <algorithm>

#include "fz_cell.cuh"
#include "fz_device.cuh"
#include "fz_kernels.h"
#include "fz_pair.cuh"

namespace fz {

namespace {

constexpr int DROWS = 4;  // warps (rows, or row chunks of a planar room) per CTA
constexpr int DCELLS = DIRECT_CELLS;  // cells of a row a warp updates

template <class R, int STAGE, bool DIM2, int KM, int LM>
__device__ __forceinline__ void direct_body(const StageArgs<R>& A, const BandArgs<R>& B, const DirectArgs& D, int bx,
                                            int by, int bz) {
  typedef typename Pair<R>::T P;
  typedef Sweep<R> Sw;
  typedef typename Sw::X X;
  const int lane = threadIdx.x;
  const int i = GHOST - 1 + bx * DCELLS + lane;
  const int il = min(i, A.Nx - GHOST);  // lanes past the room's end load its last halo centre's column
  const int member = bz / D.chunks, chunk = bz - member * D.chunks;
  const int kz = member * A.Nz;  // this member's first plane
  int j, m0, m1;                 // row (3D), march range
  if (STAGE == 0 && A.rec_n > 0 && bx == 0 && by == 0 && bz == 0)
    stage_receivers<R>(A, (int)threadIdx.y * 32 + lane, 32 * DROWS);
  if (!DIM2) {
    j = GHOST + by * DROWS + threadIdx.y;
    m0 = GHOST + chunk * D.depth;
    m1 = min(m0 + D.depth, A.Nz - GHOST);
    if (j >= A.Ny - GHOST) return;
  } else {
    j = 0;
    m0 = GHOST + (by * DROWS + (int)threadIdx.y) * D.depth;
    m1 = min(m0 + D.depth, A.Ny - GHOST);
  }
  if (m0 >= m1) return;
  const bool own = lane >= 1 && lane <= DCELLS && i < A.Nx - GHOST;
  const int64_t Sx = A.Sx, ms = DIM2 ? A.Sx : A.plane;  // stride along the march
  int64_t g = DIM2 ? XOFF + il + Sx * (int64_t)m0 + A.plane * (int64_t)(kz + GHOST)
                   : XOFF + il + Sx * (int64_t)j + A.plane * (int64_t)(kz + m0);
  const R* const qi = DIM2 ? A.vi : A.wi;  // velocity along the march
  auto ld = [&](const R* f, int64_t x) -> R { return fz_inb(A.err, x, A.nfield) ? __ldg(f + x) : R(0); };
  auto ldq = [&](int64_t x) -> P { return pmk(ld(A.pi, x), ld(qi, x)); };

  // march queue: centres m0-1 and m0, then one centre ahead per cell
  P qa, qb, qc, qd;
  X mlo, m_below, mhi;  // lo of centre m; planar rooms: lo of m - 1 and hi of m as well
  typename Sw::F Fm_lo;
  {
    const P z0 = ldq(g - 3 * ms), z1 = ldq(g - 2 * ms), z2 = ldq(g - ms), z3 = ldq(g), z4 = ldq(g + ms);
    const P z5 = ldq(g + 2 * ms);
    X lo, hi, unused;
    Sw::template centre<WENO_LO>(A, z0, z1, z2, z3, z4, lo, unused);
    Sw::centre(A, z1, z2, z3, z4, z5, mlo, hi);
    Fm_lo = Sw::face(A, lo, hi);
    m_below = lo;
    mhi = hi;
    qa = z2; qb = z3; qc = z4; qd = z5;
  }
  for (int m = m0; m < m1; ++m, g += ms) {
    const int jj = DIM2 ? m : j, k = kz + (DIM2 ? GHOST : m);
    // ---- loads of this cell
    const P qe = ldq(g + 3 * ms);
    const bool here = own && fz_inb(A.err, g, A.nfield);
    const uint8_t cls = here ? __ldg(A.cls + g) : (uint8_t)0;
    const int b = (KM >= 0 && here) ? __ldg(D.bidx + g) : -1;
    P x[5];
#pragma unroll
    for (int o = 0; o < 5; o++) x[o] = o == 2 ? pmk(qb.x, ld(A.ui, g)) : pmk(ld(A.pi, g + o - 2), ld(A.ui, g + o - 2));
    P y[7];
    if (!DIM2) {
#pragma unroll
      for (int o = 0; o < 7; o++)
        y[o] = o == 3 ? pmk(qb.x, ld(A.vi, g)) : pmk(ld(A.pi, g + (o - 3) * Sx), ld(A.vi, g + (o - 3) * Sx));
    }
    R bp = R(0), bu = R(0), bv = R(0), bw = R(0);
    if (STAGE > 0) {
      bp = ld(A.pb, g);
      bu = ld(A.ub, g);
      bv = ld(A.vb, g);
      bw = ld(A.wb, g);
    }
    const R w_in = DIM2 ? ld(A.wi, g) : qb.y;
    const R v_in = DIM2 ? qb.y : y[3].y;
    int4 rc = make_int4(0, 0, 0, 0);
    if (KM >= 0 && b >= 0) rc = __ldg(B.rec + b);

    // ---- centres
    X mlo_up, mhi_up, xlo, xhi;
    Sw::centre(A, qa, qb, qc, qd, qe, mlo_up, mhi_up);
    const typename Sw::F Fm_hi = Sw::face(A, mlo, mhi_up);
    Sw::centre(A, x[0], x[1], x[2], x[3], x[4], xlo, xhi);
    const X xlo_below = shfl_up1(xlo), xhi_above = shfl_down1(xhi);
    X ylo_below, ylo, yhi, yhi_above;
    if (!DIM2) {
      X unused;
      Sw::template centre<WENO_LO>(A, y[0], y[1], y[2], y[3], y[4], ylo_below, unused);
      Sw::centre(A, y[1], y[2], y[3], y[4], y[5], ylo, yhi);
      Sw::template centre<WENO_HI>(A, y[2], y[3], y[4], y[5], y[6], unused, yhi_above);
    }

    // ---- the cell's update, as in the marching kernel: stage combination, cPML, sources, band
    if (cls & (CLS_UPDATE | CLS_SOURCE | CLS_BAND)) {
      R pn, un, vn, wn;
      if (cls & CLS_UPDATE) {
        const P Dx = Sw::across(A, xlo_below, xhi, xlo, xhi_above);
        // a planar room's march is its y sweep; the marching kernel takes y differences from the states
        const P Dm = DIM2 ? P() : Sw::across(Fm_lo, Fm_hi);
        P Dy, Dz;
        if (DIM2) {
          Dy = Sw::across(A, m_below, mhi, mlo, mhi_up);
          Dz = pmk(R(0), R(0));
        } else {
          Dy = Sw::across(A, ylo_below, yhi, ylo, yhi_above);
          Dz = Dm;
        }
        pn = fma(A.dt_p, (Dx.x + Dy.x) + Dz.x, qb.x);
        un = fma(A.dt_v, Dx.y, x[2].y);
        vn = fma(A.dt_v, Dy.y, v_in);
        wn = fma(A.dt_v, Dz.y, w_in);
        if (STAGE > 0) {
          const R wb = (STAGE == 1) ? R(0.25) : R(2.0 / 3.0);
          pn = fma(wb, pn - bp, bp);
          un = fma(wb, un - bu, bu);
          vn = fma(wb, vn - bv, bv);
          wn = fma(wb, wn - bw, bw);
        }
        // layers by index: no coefficient is read where there is none
        const int kl = DIM2 ? GHOST : m;
        if (A.pml_on && (i < A.pml_lo[0] || i >= A.pml_hi[0] || jj < A.pml_lo[1] || jj >= A.pml_hi[1] ||
                         kl < A.pml_lo[2] || kl >= A.pml_hi[2]) && fz_inb(A.err, k, A.npc[2])) {
          const PmlCoef<R> cx = A.pcx[i], cy = A.pcy[jj], cz = A.pcz[k];
          pml_update<R, STAGE>(A, i, jj, k, cx, cy, cz, Dx, Dy, Dz, pn, un, vn, wn);
        }
        if (cls & CLS_SOURCE) pn += source_sum(A, g);
      } else {
        // a skipped cell keeps its stale output, to which a source adds and which the band replaces
        pn = A.po[g];
        if (cls & CLS_SOURCE) pn += source_sum(A, g);
        if (KM >= 0 && b >= 0) {
          un = A.uo[g];
          vn = A.vo[g];
          wn = A.wo[g];
        }
      }
      if (KM >= 0 && b >= 0 && band_inb(B, g, rc))
        band_cell<R, STAGE, KM < 0 ? 0 : KM, LM, true>(B, b, g, rc, pn, un, vn, wn);
      A.po[g] = pn;
      if ((cls & CLS_UPDATE) || (KM >= 0 && b >= 0)) {
        A.uo[g] = un;
        A.vo[g] = vn;
        A.wo[g] = wn;
      }
    }
    Fm_lo = Fm_hi;
    if (DIM2) {
      m_below = mlo;
      mhi = mhi_up;
    }
    mlo = mlo_up;
    qa = qb;
    qb = qc;
    qc = qd;
    qd = qe;
  }
}

// KM, LM: the band kernel's pole forms (2, 4, 0 = any), -1 without a band.
template <class R, int STAGE, bool DIM2, int KM>
__global__ void __launch_bounds__(32 * DROWS, 4)
    k_stage_direct(const __grid_constant__ StageArgs<R> A, const __grid_constant__ BandArgs<R> B,
                   const __grid_constant__ DirectArgs D) {
  direct_body<R, STAGE, DIM2, KM, KM < 0 ? 0 : KM>(A, B, D, blockIdx.x, blockIdx.y, blockIdx.z);
}

template <class R, int STAGE, bool DIM2>
cudaError_t launch(int fit, const StageArgs<R>& a, const BandArgs<R>& b, const DirectArgs& d, dim3 grid,
                   cudaStream_t s) {
  const dim3 block(32, DROWS, 1);
  if (fit == 2)
    k_stage_direct<R, STAGE, DIM2, 2><<<grid, block, 0, s>>>(a, b, d);
  else if (fit == 4)
    k_stage_direct<R, STAGE, DIM2, 4><<<grid, block, 0, s>>>(a, b, d);
  else if (fit == 0)
    k_stage_direct<R, STAGE, DIM2, 0><<<grid, block, 0, s>>>(a, b, d);
  else
    k_stage_direct<R, STAGE, DIM2, -1><<<grid, block, 0, s>>>(a, b, d);
  return cudaGetLastError();
}

}  // namespace

DirectShape direct_shape(int Nx, int Ny, int Nz, int nb, bool two_d, int nsm) {
  DirectShape sh;
  const int ex = Nx - 2 * GHOST, ey = Ny - 2 * GHOST, ez = Nz - 2 * GHOST;
  const int tiles = (ex + DCELLS - 1) / DCELLS;
  // a planar march of one row pays for two extra centres (of 4), so it takes two rows as soon as the warps
  // keep every scheduler busy without it. 3D rooms of so many warps run the marching kernel: their marches
  // are of one plane (compiled without the loop, the 3D form takes 17.2 instead of 16.0 us a step of 26 x 22
  // x 18 cells, 28.0 instead of 26.5 of 45 x 38 x 29 FP64: 128 registers in every instance, and other spills)
  sh.depth = two_d && ey > 1 && (int64_t)tiles * nb * ey >= 32 * (int64_t)nsm ? 2 : 1;
  sh.chunks = two_d ? 1 : ez;
  const int warps_y = (ey + sh.depth - 1) / sh.depth;
  sh.grid = dim3((unsigned)tiles, (unsigned)((warps_y + DROWS - 1) / DROWS), (unsigned)(sh.chunks * nb));
  return sh;
}

template <class R>
cudaError_t launch_stage_direct(int stage, bool two_d, const StageArgs<R>& a, const BandArgs<R>& b,
                                const DirectArgs& d, dim3 grid, cudaStream_t s) {
  const int fit = b.nB <= 0 ? -1 : (b.K <= 2 && b.L <= 2) ? 2 : (b.K <= 4 && b.L <= 4) ? 4 : 0;
  if (!two_d) {
    if (stage == 0) return launch<R, 0, false>(fit, a, b, d, grid, s);
    if (stage == 1) return launch<R, 1, false>(fit, a, b, d, grid, s);
    return launch<R, 2, false>(fit, a, b, d, grid, s);
  }
  if (stage == 0) return launch<R, 0, true>(fit, a, b, d, grid, s);
  if (stage == 1) return launch<R, 1, true>(fit, a, b, d, grid, s);
  return launch<R, 2, true>(fit, a, b, d, grid, s);
}

template cudaError_t launch_stage_direct<float>(int, bool, const StageArgs<float>&, const BandArgs<float>&,
                                                const DirectArgs&, dim3, cudaStream_t);
template cudaError_t launch_stage_direct<double>(int, bool, const StageArgs<double>&, const BandArgs<double>&,
                                                 const DirectArgs&, dim3, cudaStream_t);

}  // namespace fz
