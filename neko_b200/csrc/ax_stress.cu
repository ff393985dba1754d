// ax_stress.cu -- the full-stress Helmholtz operator of the velocity solve
// with variable viscosity (ax_helm_full_t%compute_vector,
// src/math/bcknd/device/ax_helm_full_device.F90:190-259; CPU form
// src/math/bcknd/cpu/ax_helm_full_cpu.f90:181-375; device kernel
// src/math/bcknd/device/cuda/ax_helm_full_kernel.h):
//
//   per point, with C the cofactor matrix (C = jac * d(r,s,t)/d(x,y,z)),
//   G_c = C^T (d/dr, d/ds, d/dt) u_c            (jac * physical gradient)
//   S   = h1 w3 / jac * (G + G^T)                (symmetric, 6 values)
//   F_c = C S_c                                  (flux of component c)
//   A u_c = D_r^T F_c,r + D_s^T F_c,s + D_t^T F_c,t
//
// and the h2 B term (cuda_ax_helm_stress_vector_part2).
//
// B200 form: a persistent streaming kernel (lx 4, 6, 8, 10) -- the three
// components, h1, 1/jac and the nine cofactors of an element (14 arrays)
// arrive in one bulk-copy stage, the strain is formed once for the three
// components, the nine flux planes are written over the cofactors in the
// stage and the transposed contractions read them back.  112 B of
// coefficients and 48 B of fields per point: 136 B per point moved (17 arrays
// of 8 B).  At lx 8 the contractions run on the FP64 tensor instructions
// (ax_stress_mma_kernel).  Other orders, and operands off a 16-byte boundary,
// use a general kernel (one element per block, fluxes kept in registers).
#include <cstdint>
#include <cstdio>
#include <cstdlib>

#include "nb_chain.cuh"
#include "nb_kernels.h"
#include "nb_precond.h"
#include "nb_problem.h"
#include "nb_reduce.cuh"
#include "nb_tma.cuh"

namespace nb {

struct StressIo {
  double *out[3];
  const double *in[3];
};
// h1, 1/jac, cofactors drdx, drdy, drdz, dsdx, dsdy, dsdz, dtdx, dtdy, dtdz
struct StressGeo {
  const double *h1, *jacinv, *c[9];
};

// The CG step folded into the operator (coupled CG): p_c = z_c + beta p_c
// formed from the stage and stored, the operator applied to the new p, and
// pap = sum over local points of p . w with alpha = rtz / pap.  p is zero on
// masked points (z is) and continuous, so the local sum equals the
// mult-weighted one after the gather-scatter and mask.
struct StressCg {
  const double *z[3] = {nullptr, nullptr, nullptr};
  double *pout[3] = {nullptr, nullptr, nullptr};
  CgState *st = nullptr;
  double *partials = nullptr;
  unsigned *counter = nullptr;
};

// Strain and fluxes at one point: g[c][0..2] = (d/dr, d/ds, d/dt) of
// component c, f[c][0..2] = (r, s, t) fluxes.  The order of the operations
// follows the reference kernel (ax_helm_full_kernel.h).
__device__ __forceinline__ void stress_point(const double g[3][3], const double cf[9],
                                             double dj, double f[3][3]) {
  const double rx = cf[0], ry = cf[1], rz = cf[2], sx = cf[3], sy = cf[4], sz = cf[5],
               tx = cf[6], ty = cf[7], tz = cf[8];
  double G[3][3];
#pragma unroll
  for (int c = 0; c < 3; c++) {
    G[c][0] = g[c][0] * rx + g[c][1] * sx + g[c][2] * tx;
    G[c][1] = g[c][0] * ry + g[c][1] * sy + g[c][2] * ty;
    G[c][2] = g[c][0] * rz + g[c][1] * sz + g[c][2] * tz;
  }
  const double s11 = dj * (G[0][0] + G[0][0]);
  const double s22 = dj * (G[1][1] + G[1][1]);
  const double s33 = dj * (G[2][2] + G[2][2]);
  const double s12 = dj * (G[0][1] + G[1][0]);
  const double s13 = dj * (G[0][2] + G[2][0]);
  const double s23 = dj * (G[1][2] + G[2][1]);
  const double S[3][3] = {{s11, s12, s13}, {s12, s22, s23}, {s13, s23, s33}};
#pragma unroll
  for (int c = 0; c < 3; c++) {
    f[c][0] = rx * S[c][0] + ry * S[c][1] + rz * S[c][2];
    f[c][1] = sx * S[c][0] + sy * S[c][1] + sz * S[c][2];
    f[c][2] = tx * S[c][0] + ty * S[c][1] + tz * S[c][2];
  }
}

// ---------------------------------------------------------------------------
// Streaming kernel (lx 4, 6, 10; lx 8 below).  Bound by HBM (136 B a point, 152 with
// h2; 184 / 200 in the CG form) with shared-memory wavefronts close behind.
//
// The nine flux planes lie over the nine cofactor arrays of the element's own
// stage: a thread reads the nine cofactors of a point and writes that point's
// nine fluxes over them, and no thread reads another point's cofactors.  So
// a stage is all the memory an element needs (14 arrays) and two stages of
// lx 10 (224 KB) fit a multiprocessor.  With separate planes lx 10 had no
// streaming form (272 us on 2.2 M points, plus 29 us for the h2 term; 141 us
// in this one).  h2, B and (CG form) z go straight to registers instead of
// staging up to five more arrays; they are brought to L2 when the stage is
// filled.
// Registers (512 threads a multiprocessor: 128 each) hold two rows of D at a
// time at lx 10, reloaded for the second pass, and the components are
// differentiated one after the other.  At lx 4 and 6 the four rows fit and are
// loaded once (HOLD): 76 against 92 us on 3.0 M points at lx 4, 101 against 113 at
// lx 6 (84 and 99, 107 and 121 with h2).
// ---------------------------------------------------------------------------
template <int LX, int S, int KS>
struct StressCfg {
  static constexpr int L2 = LX * LX, L3 = L2 * LX, NA = 14;
  static constexpr int THREADS = ((L2 * KS + 31) / 32) * 32;
  static constexpr size_t ABYTES = (size_t)L3 * sizeof(double);
  static constexpr size_t SMEM = S * NA * ABYTES + L2 * sizeof(double) + 16 * S;
  static constexpr int BLOCKS0 = (int)(233472 / (SMEM + 1024 + 128));
  static constexpr int BLOCKS1 = BLOCKS0 * THREADS > 512 ? 512 / THREADS : BLOCKS0;
  static constexpr int BLOCKS = BLOCKS1 < 1 ? 1 : BLOCKS1;
  static constexpr bool HOLD = LX <= 6;
};

template <int LX, int S, int KS, bool CG>
__global__ void __launch_bounds__(StressCfg<LX, S, KS>::THREADS, StressCfg<LX, S, KS>::BLOCKS)
    ax_stress_tma_kernel(StressIo io, StressGeo geo, const double *__restrict__ dx,
                         const double *__restrict__ dy, const double *__restrict__ dz,
                         const double *__restrict__ w3, const double *__restrict__ h2,
                         const double *__restrict__ Bm, const int nelv, int *__restrict__ err,
                         const int *__restrict__ skip, StressCg cg) {
  using C = StressCfg<LX, S, KS>;
  constexpr int L2 = C::L2, L3 = C::L3, NA = C::NA, KP = LX / KS;
  static_assert(LX % KS == 0 && LX % 2 == 0, "k split must divide an even lx");
  extern __shared__ __align__(128) unsigned char smem_stress[];
  double *stage = reinterpret_cast<double *>(smem_stress);
  double *sDz = stage + S * NA * L3;
  uint64_t *full = reinterpret_cast<uint64_t *>(sDz + L2);

  const int tid = threadIdx.x;
  const int G = gridDim.x, b = blockIdx.x;
  const int nt = b < nelv ? (nelv - b + G - 1) / G : 0;
  if (tid == 0) {
    for (int s = 0; s < S; s++) mbar_init(&full[s], 1);
    fence_barrier_init();
  }
  chain();
  if (skip && *skip) return;
  if (CG && cg.st->done) return;
  const double beta = CG ? cg.st->beta : 0.0;
  for (int q = tid; q < L2; q += C::THREADS) sDz[q] = dz[q];
  __syncthreads();
  // stage slot: u, v, w (the old directions in the CG form), h1, 1/jac, the
  // nine cofactors
  auto issue = [&](int t, int s) {
    const long e = b + (long)t * G;
    mbar_arrive_expect_tx(&full[s], (uint32_t)(NA * C::ABYTES));
#pragma unroll
    for (int a = 0; a < NA; a++) {
      const double *src =
          a < 3 ? io.in[a] : (a == 3 ? geo.h1 : (a == 4 ? geo.jacinv : geo.c[a - 5]));
      bulk_g2s(stage + (size_t)(s * NA + a) * L3, src + e * L3, (uint32_t)C::ABYTES, &full[s]);
    }
    // operands that go to registers, to L2 meanwhile
    if (h2) {
      bulk_prefetch_l2(h2 + e * L3, (uint32_t)C::ABYTES);
      bulk_prefetch_l2(Bm + e * L3, (uint32_t)C::ABYTES);
    }
    if constexpr (CG) {
#pragma unroll
      for (int c = 0; c < 3; c++) bulk_prefetch_l2(cg.z[c] + e * L3, (uint32_t)C::ABYTES);
    }
  };
  if (tid == 0)
    for (int t = 0; t < S && t < nt; t++) issue(t, t);

  const bool act = tid < L2 * KS;
  const int col = tid % L2, kh = tid / L2;
  const int i = col % LX, j = col / LX, k0 = kh * KP;

  // rows of the derivative matrices: dx(i, l), dy(j, l), then dx(l, i), dy(l, j)
  double Dxi[LX], Dyj[LX], Dxti[LX], Dytj[LX];
  auto rows = [&] {
#pragma unroll
    for (int l = 0; l < LX; l++) {
      Dxi[l] = __ldg(dx + i + LX * l);
      Dyj[l] = __ldg(dy + j + LX * l);
    }
  };
  auto rows_t = [&] {
#pragma unroll
    for (int l = 0; l < LX; l++) {
      Dxti[l] = __ldg(dx + l + LX * i);
      Dytj[l] = __ldg(dy + l + LX * j);
    }
  };
  if (C::HOLD) {
    rows();
    rows_t();
  }

  int t = 0;
  bool failed = false;
  double pap = 0.0;
  for (; t < nt; t++) {
    const int s = t % S;
    const long e = b + (long)t * G;
    double *slot = stage + (size_t)s * NA * L3;
    double *planes = slot + 5 * L3;  // fluxes: component-major, (r, s, t)
    // global operands of this thread's points, in flight during the wait
    double hb[KP], zc[CG ? 3 : 1][KP];
    if (act) {
#pragma unroll
      for (int kk = 0; kk < KP; kk++) {
        const long g = e * L3 + col + L2 * (k0 + kk);
        hb[kk] = h2 ? __ldg(h2 + g) * __ldg(Bm + g) : 0.0;
        if constexpr (CG) {
#pragma unroll
          for (int c = 0; c < 3; c++) zc[c][kk] = __ldg(cg.z[c] + g);
        }
      }
    }
    const bool ok = mbar_wait(&full[s], (uint32_t)((t / S) & 1));
    if (__syncthreads_or(!ok)) {
      failed = true;
      break;
    }
    if constexpr (CG) {  // p = z + beta p for this thread's points, in the stage and stored
      if (act) {
#pragma unroll
        for (int c = 0; c < 3; c++)
#pragma unroll
          for (int kk = 0; kk < KP; kk++) {
            const int q = col + L2 * (k0 + kk);
            const double pn = zc[c][kk] + beta * slot[c * L3 + q];
            slot[c * L3 + q] = pn;
            cg.pout[c][e * L3 + q] = pn;
          }
      }
      __syncthreads();  // the element's new directions complete in the stage
    }
    if (act) {
      if (!C::HOLD) rows();
      double g[KP][3][3];
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const double *su = slot + c * L3;
        double cu[LX];  // this thread's (i, j) column
#pragma unroll
        for (int l = 0; l < LX; l++) cu[l] = su[col + L2 * l];
#pragma unroll
        for (int kk = 0; kk < KP; kk++) {
          const int k = k0 + kk;
          const double2 *row = reinterpret_cast<const double2 *>(su + LX * j + L2 * k);
          double ur = 0, us = 0, ut = 0;
#pragma unroll
          for (int l = 0; l < LX; l += 2) {
            const double2 v = row[l / 2];
            ur += Dxi[l] * v.x;
            us += Dyj[l] * su[i + LX * l + L2 * k];
            ut += sDz[k + LX * l] * cu[l];
            ur += Dxi[l + 1] * v.y;
            us += Dyj[l + 1] * su[i + LX * (l + 1) + L2 * k];
            ut += sDz[k + LX * (l + 1)] * cu[l + 1];
          }
          g[kk][c][0] = ur;
          g[kk][c][1] = us;
          g[kk][c][2] = ut;
        }
      }
#pragma unroll
      for (int kk = 0; kk < KP; kk++) {
        const int p = col + L2 * (k0 + kk);
        double cf[9];
#pragma unroll
        for (int a = 0; a < 9; a++) cf[a] = planes[a * L3 + p];
        const double dj = slot[3 * L3 + p] * __ldg(w3 + p) * slot[4 * L3 + p];
        double f[3][3];
        stress_point(g[kk], cf, dj, f);
#pragma unroll
        for (int c = 0; c < 3; c++)
#pragma unroll
          for (int d = 0; d < 3; d++) planes[(3 * c + d) * L3 + p] = f[c][d];
      }
    }
    __syncthreads();  // flux planes complete
    if (act) {
      if (!C::HOLD) rows_t();
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const double *fr = planes + (3 * c) * L3, *fs = fr + L3, *ft = fs + L3;
        double rt[LX];
#pragma unroll
        for (int l = 0; l < LX; l++) rt[l] = ft[col + L2 * l];
        double *wo = io.out[c];
#pragma unroll
        for (int kk = 0; kk < KP; kk++) {
          const int k = k0 + kk;
          const double2 *row = reinterpret_cast<const double2 *>(fr + LX * j + L2 * k);
          const double2 *dk = reinterpret_cast<const double2 *>(sDz + LX * k);
          double a = 0, cc = 0, d = 0;
#pragma unroll
          for (int l = 0; l < LX; l += 2) {
            const double2 v = row[l / 2], z = dk[l / 2];
            a += Dxti[l] * v.x;
            cc += Dytj[l] * fs[i + LX * l + L2 * k];
            d += z.x * rt[l];
            a += Dxti[l + 1] * v.y;
            cc += Dytj[l + 1] * fs[i + LX * (l + 1) + L2 * k];
            d += z.y * rt[l + 1];
          }
          const int q = col + L2 * k;
          const double u = slot[c * L3 + q];
          double v = a + cc + d;
          if (h2) v = v + hb[kk] * u;  // au + h2 B u, the part2 order
          wo[e * L3 + q] = v;
          if (CG) pap += u * v;
        }
      }
    }
    // this thread's writes to the stage come before the next copy into it
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();  // stage s consumed
    if (tid == 0 && t + S < nt) issue(t + S, s);
  }
  if (failed) {
    if (tid == 0) {
      atomicExch(err, 1);
      // bounded wait for this CTA's copies still in flight
      for (int q = t; q < nt && q < t + S; q++) mbar_wait(&full[q % S], (uint32_t)((q / S) & 1));
    }
    __syncthreads();
  }
  if constexpr (CG) {
    double tot;  // every block takes part, a failed one with its partial sum
    if (grid_sum<C::THREADS>(pap, cg.partials, cg.counter, &tot)) {
      cg.st->pap = tot;
      cg.st->alpha = cg.st->rtz1 / tot;
    }
  }
}

// ---------------------------------------------------------------------------
// lx = 8: the contractions within a k-plane on the FP64 matrix instruction.
// An 8 x 8 plane is one m8n8k4 tile (two k-steps), with no padding.  The
// kernel above is bound by shared-memory wavefronts (about 330 a warp of
// points: an r or s derivative reads eight values a point, each load two
// wavefronts); here a lane owns the points (j, i) = (lane / 4, 2 (lane % 4) +
// {0, 1}) of a plane, the tile's result layout, and
//   r derivative: A = the plane itself, its fragment the lane's own values
//                 (the contraction index taken as 2 t + s in k-step s);
//   s derivative: B = the plane, two loads a lane;
//   r flux:       A = the flux, straight from the lane's registers;
//   s flux:       through the warp's own plane of the stage, warp-synchronous;
//   t:            plain FMAs down the lane's column, 16-byte loads.
// About 95 wavefronts a warp of points (132 measured, with the copies into the
// stage and 18 of conflicts).  Four warps an element, two planes each.  The matrix instruction runs at the FP64 FMA rate (37 against 33
// TFLOP/s measured), so it saves the operand traffic, not arithmetic.
// A fused step on 3 x 2.1 M points: 78 us, 104 with the kernel above.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void mma_f64(double (&c)[2], double a, double b) {
  asm volatile(
      "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}

struct StressMma {
  static constexpr int LX = 8, L2 = 64, L3 = 512, NA = 14, S = 2, THREADS = 128;
  static constexpr size_t ABYTES = L3 * sizeof(double);
  static constexpr size_t SMEM = S * NA * ABYTES + L2 * sizeof(double) + 16 * S;
};

// OUT2: results start on 16-byte boundaries and are stored in pairs.
template <bool CG, bool OUT2>
__global__ void __launch_bounds__(StressMma::THREADS, 2)
    ax_stress_mma_kernel(StressIo io, StressGeo geo, const double *__restrict__ dx,
                         const double *__restrict__ dy, const double *__restrict__ dz,
                         const double *__restrict__ w3, const double *__restrict__ h2,
                         const double *__restrict__ Bm, const int nelv, int *__restrict__ err,
                         const int *__restrict__ skip, StressCg cg) {
  using C = StressMma;
  constexpr int LX = C::LX, L2 = C::L2, L3 = C::L3, NA = C::NA, S = C::S;
  extern __shared__ __align__(128) unsigned char smem_stress[];
  double *stage = reinterpret_cast<double *>(smem_stress);
  double *sDz = stage + S * NA * L3;
  uint64_t *full = reinterpret_cast<uint64_t *>(sDz + L2);

  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int G = gridDim.x, b = blockIdx.x;
  const int nt = b < nelv ? (nelv - b + G - 1) / G : 0;
  if (tid == 0) {
    for (int s = 0; s < S; s++) mbar_init(&full[s], 1);
    fence_barrier_init();
  }
  chain();
  if (skip && *skip) return;
  if (CG && cg.st->done) return;
  const double beta = CG ? cg.st->beta : 0.0;
  for (int q = tid; q < L2; q += C::THREADS) sDz[q] = dz[q];
  __syncthreads();
  auto issue = [&](int t, int s) {
    const long e = b + (long)t * G;
    mbar_arrive_expect_tx(&full[s], (uint32_t)(NA * C::ABYTES));
#pragma unroll
    for (int a = 0; a < NA; a++) {
      const double *src =
          a < 3 ? io.in[a] : (a == 3 ? geo.h1 : (a == 4 ? geo.jacinv : geo.c[a - 5]));
      bulk_g2s(stage + (size_t)(s * NA + a) * L3, src + e * L3, (uint32_t)C::ABYTES, &full[s]);
    }
    if (h2) {
      bulk_prefetch_l2(h2 + e * L3, (uint32_t)C::ABYTES);
      bulk_prefetch_l2(Bm + e * L3, (uint32_t)C::ABYTES);
    }
    if constexpr (CG) {
#pragma unroll
      for (int c = 0; c < 3; c++) bulk_prefetch_l2(cg.z[c] + e * L3, (uint32_t)C::ABYTES);
    }
  };
  if (tid == 0)
    for (int t = 0; t < S && t < nt; t++) issue(t, t);

  // tile coordinates: row m, column pair n
  const int m = lane >> 2, n = lane & 3, k0 = 2 * wid;
  const int own = LX * m + 2 * n;  // the lane's two points in a plane
  // fragments of D: r derivative (B), s derivative (A), r flux (B), s flux (A)
  double dr[2], ds[2], fr[2], fs[2];
#pragma unroll
  for (int s = 0; s < 2; s++) {
    dr[s] = __ldg(dx + m + LX * (2 * n + s));
    ds[s] = __ldg(dy + m + LX * (n + 4 * s));
    fr[s] = __ldg(dx + (2 * n + s) + LX * m);
    fs[s] = __ldg(dy + (n + 4 * s) + LX * m);
  }
  auto get2 = [](const double *p, double (&v)[2]) {
    const double2 t = *reinterpret_cast<const double2 *>(p);
    v[0] = t.x;
    v[1] = t.y;
  };
  auto put2 = [](double *p, const double (&v)[2]) {
    *reinterpret_cast<double2 *>(p) = make_double2(v[0], v[1]);
  };

  int t = 0;
  bool failed = false;
  double pap = 0.0;
  for (; t < nt; t++) {
    const int s = t % S;
    const long e = b + (long)t * G;
    double *slot = stage + (size_t)s * NA * L3;
    const bool ok = mbar_wait(&full[s], (uint32_t)((t / S) & 1));
    if (__syncthreads_or(!ok)) {
      failed = true;
      break;
    }
    if constexpr (CG) {  // p = z + beta p for the lane's points, in the stage and stored
#pragma unroll
      for (int c = 0; c < 3; c++)
#pragma unroll
        for (int kk = 0; kk < 2; kk++) {
          const int q = L2 * (k0 + kk) + own;
          const double2 z = __ldg(reinterpret_cast<const double2 *>(cg.z[c] + e * L3 + q));
          double p[2];
          get2(slot + c * L3 + q, p);
          p[0] = z.x + beta * p[0];
          p[1] = z.y + beta * p[1];
          put2(slot + c * L3 + q, p);
          put2(cg.pout[c] + e * L3 + q, p);
        }
      __syncthreads();  // the element's new directions complete in the stage
    }
    // t derivatives of both planes, down the lane's column
    double ut[2][3][2];
#pragma unroll
    for (int c = 0; c < 3; c++) {
#pragma unroll
      for (int kk = 0; kk < 2; kk++) ut[kk][c][0] = ut[kk][c][1] = 0.0;
#pragma unroll
      for (int l = 0; l < LX; l++) {
        double v[2];
        get2(slot + c * L3 + L2 * l + own, v);
#pragma unroll
        for (int kk = 0; kk < 2; kk++) {
          const double d = sDz[k0 + kk + LX * l];
          ut[kk][c][0] += d * v[0];
          ut[kk][c][1] += d * v[1];
        }
      }
    }
    double acc[2][3][2];  // r and s flux divergence at the lane's points
#pragma unroll
    for (int kk = 0; kk < 2; kk++) {
      const int base = L2 * (k0 + kk);
      double g[2][3][3];
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const double *u = slot + c * L3 + base;
        double v[2], ur[2] = {0.0, 0.0}, us[2] = {0.0, 0.0};
        get2(u + own, v);
#pragma unroll
        for (int h = 0; h < 2; h++) mma_f64(ur, v[h], dr[h]);
#pragma unroll
        for (int h = 0; h < 2; h++) mma_f64(us, ds[h], u[LX * (n + 4 * h) + m]);
#pragma unroll
        for (int h = 0; h < 2; h++) {
          g[h][c][0] = ur[h];
          g[h][c][1] = us[h];
          g[h][c][2] = ut[kk][c][h];
        }
      }
      double cf[2][9], hv[2], jv[2], f[2][3][3];
#pragma unroll
      for (int a = 0; a < 9; a++) {
        double v[2];
        get2(slot + (5 + a) * L3 + base + own, v);
        cf[0][a] = v[0];
        cf[1][a] = v[1];
      }
      get2(slot + 3 * L3 + base + own, hv);
      get2(slot + 4 * L3 + base + own, jv);
      const double2 wv = make_double2(__ldg(w3 + base + own), __ldg(w3 + base + own + 1));
      stress_point(g[0], cf[0], hv[0] * wv.x * jv[0], f[0]);
      stress_point(g[1], cf[1], hv[1] * wv.y * jv[1], f[1]);
      // s and t fluxes over the cofactors just read, the lane's own points
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const double vs[2] = {f[0][c][1], f[1][c][1]}, vt[2] = {f[0][c][2], f[1][c][2]};
        put2(slot + (5 + c) * L3 + base + own, vs);
        put2(slot + (8 + c) * L3 + base + own, vt);
      }
      __syncwarp();  // the plane's s fluxes, all from this warp
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const double *v = slot + (5 + c) * L3 + base;
        acc[kk][c][0] = acc[kk][c][1] = 0.0;
#pragma unroll
        for (int h = 0; h < 2; h++) mma_f64(acc[kk][c], f[h][c][0], fr[h]);
#pragma unroll
        for (int h = 0; h < 2; h++) mma_f64(acc[kk][c], fs[h], v[LX * (n + 4 * h) + m]);
      }
    }
    __syncthreads();  // every plane's t fluxes complete
    double hb[2][2];
    if (h2) {
#pragma unroll
      for (int kk = 0; kk < 2; kk++) {
        const long q = e * L3 + L2 * (k0 + kk) + own;
        const double2 x = __ldg(reinterpret_cast<const double2 *>(h2 + q)),
                      y = __ldg(reinterpret_cast<const double2 *>(Bm + q));
        hb[kk][0] = x.x * y.x;
        hb[kk][1] = x.y * y.y;
      }
    }
#pragma unroll
    for (int c = 0; c < 3; c++) {
      double d[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
#pragma unroll
      for (int l = 0; l < LX; l++) {
        double v[2];
        get2(slot + (8 + c) * L3 + L2 * l + own, v);
#pragma unroll
        for (int kk = 0; kk < 2; kk++) {
          const double z = sDz[l + LX * (k0 + kk)];
          d[kk][0] += z * v[0];
          d[kk][1] += z * v[1];
        }
      }
#pragma unroll
      for (int kk = 0; kk < 2; kk++) {
        const int q = L2 * (k0 + kk) + own;
        double u[2], v[2];
        get2(slot + c * L3 + q, u);
#pragma unroll
        for (int h = 0; h < 2; h++) {
          v[h] = acc[kk][c][h] + d[kk][h];
          if (h2) v[h] = v[h] + hb[kk][h] * u[h];  // au + h2 B u, the part2 order
          if (CG) pap += u[h] * v[h];
        }
        if constexpr (OUT2) {
          put2(io.out[c] + e * L3 + q, v);
        } else {
          io.out[c][e * L3 + q] = v[0];
          io.out[c][e * L3 + q + 1] = v[1];
        }
      }
    }
    // this thread's writes to the stage come before the next copy into it
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();  // stage s consumed
    if (tid == 0 && t + S < nt) issue(t + S, s);
  }
  if (failed) {
    if (tid == 0) {
      atomicExch(err, 1);
      // bounded wait for this CTA's copies still in flight
      for (int q = t; q < nt && q < t + S; q++) mbar_wait(&full[q % S], (uint32_t)((q / S) & 1));
    }
    __syncthreads();
  }
  if constexpr (CG) {
    double tot;  // every block takes part, a failed one with its partial sum
    if (grid_sum<C::THREADS>(pap, cg.partials, cg.counter, &tot)) {
      cg.st->pap = tot;
      cg.st->alpha = cg.st->rtz1 / tot;
    }
  }
}

template <bool CG>
static cudaError_t launch_stress_mma(const StressIo &io, const StressGeo &geo, const double *dx,
                                     const double *dy, const double *dz, const double *w3,
                                     const double *h2, const double *Bm, int nelv,
                                     cudaStream_t st, int *err, const int *skip,
                                     const StressCg &cg = StressCg{}) {
  using C = StressMma;
  auto off = [](const void *q) { return (reinterpret_cast<uintptr_t>(q) & 15) != 0; };
  if (off(h2) || off(Bm)) return cudaErrorNotSupported;  // read in 16-byte pairs
  const bool out2 = !off(io.out[0]) && !off(io.out[1]) && !off(io.out[2]);
  auto kern = out2 ? ax_stress_mma_kernel<CG, true> : ax_stress_mma_kernel<CG, false>;
  static int grids[2][64] = {{0}};
  int(&grid_per_dev)[64] = grids[out2];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  int &g = grid_per_dev[dev & 63];
  if (g == 0) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, C::THREADS, C::SMEM);
    if (e != cudaSuccess) return e;
    g = (per_sm > 0 ? per_sm : 1) * device_sms();
  }
  if (nelv <= 0) return cudaSuccess;
  if (!err) err = dropin_error_word();
  if (!err) return cudaErrorInvalidSymbol;
  return launch_chained(3L * nelv * C::L3, kern,
                        nelv < g ? nelv : g, C::THREADS, C::SMEM, st, io, geo, dx, dy, dz,
                        w3, h2, Bm, nelv, err, skip, cg);
}

template <int LX, int S, int KS, bool CG = false>
static cudaError_t launch_stress_tma(const StressIo &io, const StressGeo &geo, const double *dx,
                                     const double *dy, const double *dz, const double *w3,
                                     const double *h2, const double *Bm, int nelv,
                                     cudaStream_t st, int *err, const int *skip,
                                     const StressCg &cg = StressCg{}) {
  using C = StressCfg<LX, S, KS>;
  auto kern = ax_stress_tma_kernel<LX, S, KS, CG>;
  static int grid_per_dev[64] = {0};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  int &g = grid_per_dev[dev & 63];
  if (g == 0) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, C::THREADS, C::SMEM);
    if (e != cudaSuccess) return e;
    g = (per_sm > 0 ? per_sm : 1) * device_sms();
  }
  if (nelv <= 0) return cudaSuccess;
  if (!err) err = dropin_error_word();
  if (!err) return cudaErrorInvalidSymbol;
  const int grid = nelv < g ? nelv : g;
  launch_chained(3L * nelv * C::L3, kern, grid, C::THREADS, C::SMEM, st, io, geo, dx, dy, dz, w3,
                 h2, Bm, nelv, err, skip, cg);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// General kernel: any lx in 2..16, one element per block at a time, KS
// threads per (i, j) column taking the planes k = kh, kh + KS, ...  Up to
// lx 12 the nine flux planes sit in shared memory beside the inputs; above
// that the fluxes of a thread's points stay in registers and pass through
// the input buffer component by component.
// ---------------------------------------------------------------------------
template <int LX>
struct StressGen {
  static constexpr int L2 = LX * LX, L3 = L2 * LX;
  static constexpr int KS = LX <= 11 ? (LX < 4 ? LX : 4) : 2;
  static constexpr int KPM = (LX + KS - 1) / KS;
  static constexpr int THREADS = L2 * KS;
  static constexpr bool PLANES = LX <= 12;
  static constexpr size_t SMEM = (size_t)((PLANES ? 13 : 4) * L3 + 3 * L2) * sizeof(double);
};

template <int LX>
__global__ void __launch_bounds__(StressGen<LX>::THREADS)
    ax_stress_gen_kernel(StressIo io, StressGeo geo, const double *__restrict__ dx,
                         const double *__restrict__ dy, const double *__restrict__ dz,
                         const double *__restrict__ w3, const int nelv,
                         const int *__restrict__ skip) {
  using C = StressGen<LX>;
  constexpr int L2 = C::L2, L3 = C::L3, KS = C::KS, KPM = C::KPM;
  if (skip && *skip) return;
  extern __shared__ __align__(16) double smem_gen[];
  double *buf = smem_gen;  // u, v, w
  double *sW3 = buf + 3 * L3;
  double *sDx = sW3 + L3, *sDy = sDx + L2, *sDz = sDy + L2;
  double *planes = C::PLANES ? sDz + L2 : buf;  // 9 planes, or one component's 3 in buf
  const int tid = threadIdx.x;
  for (int q = tid; q < L2; q += C::THREADS) {
    sDx[q] = dx[q];
    sDy[q] = dy[q];
    sDz[q] = dz[q];
  }
  for (int q = tid; q < L3; q += C::THREADS) sW3[q] = w3[q];
  const int col = tid % L2, kh = tid / L2;
  const int i = col % LX, j = col / LX;
  for (long e = blockIdx.x; e < nelv; e += gridDim.x) {
    __syncthreads();  // buffers free (and matrices loaded)
    for (int q = tid; q < 3 * L3; q += C::THREADS)
      buf[q] = io.in[q / L3][e * L3 + q % L3];
    __syncthreads();
    double f[C::PLANES ? 1 : KPM][3][3];
#pragma unroll
    for (int m = 0; m < KPM; m++) {
      const int k = kh + KS * m;
      if (k < LX) {
        const int p = col + L2 * k;
        double g[3][3];
#pragma unroll
        for (int c = 0; c < 3; c++) {
          const double *su = buf + c * L3;
          double ur = 0, us = 0, ut = 0;
#pragma unroll
          for (int l = 0; l < LX; l++) {
            ur += sDx[i + LX * l] * su[l + LX * j + L2 * k];
            us += sDy[j + LX * l] * su[i + LX * l + L2 * k];
            ut += sDz[k + LX * l] * su[col + L2 * l];
          }
          g[c][0] = ur;
          g[c][1] = us;
          g[c][2] = ut;
        }
        const long gp = e * L3 + p;
        double cf[9];
#pragma unroll
        for (int a = 0; a < 9; a++) cf[a] = __ldg(geo.c[a] + gp);
        const double dj = __ldg(geo.h1 + gp) * sW3[p] * __ldg(geo.jacinv + gp);
        if constexpr (C::PLANES) {
          double fp[3][3];
          stress_point(g, cf, dj, fp);
#pragma unroll
          for (int c = 0; c < 3; c++)
#pragma unroll
            for (int d = 0; d < 3; d++) planes[(3 * c + d) * L3 + p] = fp[c][d];
        } else {
          stress_point(g, cf, dj, f[m]);
        }
      }
    }
#pragma unroll 1
    for (int c = 0; c < 3; c++) {
      const double *fr, *fs, *ft;
      if constexpr (C::PLANES) {
        if (c == 0) __syncthreads();  // all nine planes written
        fr = planes + 3 * c * L3;
      } else {
        __syncthreads();  // inputs (or the previous component's planes) read
#pragma unroll
        for (int m = 0; m < KPM; m++) {
          const int k = kh + KS * m;
          if (k < LX)
#pragma unroll
            for (int d = 0; d < 3; d++) buf[d * L3 + col + L2 * k] = f[m][c][d];
        }
        __syncthreads();
        fr = buf;
      }
      fs = fr + L3;
      ft = fs + L3;
#pragma unroll
      for (int m = 0; m < KPM; m++) {
        const int k = kh + KS * m;
        if (k < LX) {
          double a = 0, cc = 0, d = 0;
#pragma unroll
          for (int l = 0; l < LX; l++) {
            a += sDx[l + LX * i] * fr[l + LX * j + L2 * k];
            cc += sDy[l + LX * j] * fs[i + LX * l + L2 * k];
            d += sDz[l + LX * k] * ft[col + L2 * l];
          }
          io.out[c][e * L3 + col + L2 * k] = a + cc + d;
        }
      }
    }
  }
}

template <int LX>
static cudaError_t launch_stress_gen(const StressIo &io, const StressGeo &geo, const double *dx,
                                     const double *dy, const double *dz, const double *w3,
                                     int nelv, cudaStream_t st, const int *skip) {
  using C = StressGen<LX>;
  auto kern = ax_stress_gen_kernel<LX>;
  static bool attr[64] = {false};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (!attr[dev & 63]) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
    if (e != cudaSuccess) return e;
    attr[dev & 63] = true;
  }
  if (nelv <= 0) return cudaSuccess;
  const int cap = 64 * device_sms();
  const int grid = nelv < cap ? nelv : cap;
  kern<<<grid, C::THREADS, C::SMEM, st>>>(io, geo, dx, dy, dz, w3, nelv, skip);
  return cudaGetLastError();
}

// (au, av, aw) = A_stress (u, v, w), h1 part.  The streaming kernel for lx
// 4, 6, 8, 10 with 16-byte aligned operands, the general kernel otherwise.
cudaError_t ax_stress(double *au, double *av, double *aw, const double *u, const double *v,
                      const double *w, const double *dx, const double *dy, const double *dz,
                      const double *h1, const double *jacinv, const double *const cof[9],
                      const double *w3, int nelv, int lx, cudaStream_t s, int *err,
                      const int *skip, const double *h2, const double *Bm) {
  StressIo io{{au, av, aw}, {u, v, w}};
  StressGeo geo{h1, jacinv, {cof[0], cof[1], cof[2], cof[3], cof[4], cof[5], cof[6], cof[7],
                             cof[8]}};
  bool aligned = true;
  const void *ptrs[] = {u, v, w, h1, jacinv, cof[0], cof[1], cof[2], cof[3],
                        cof[4], cof[5], cof[6], cof[7], cof[8]};
  for (const void *q : ptrs)
    if (reinterpret_cast<uintptr_t>(q) & 15) aligned = false;
  if (aligned) {
    switch (lx) {
      case 4: return launch_stress_tma<4, 3, 2>(io, geo, dx, dy, dz, w3, h2, Bm, nelv, s, err, skip);
      case 6: return launch_stress_tma<6, 2, 3>(io, geo, dx, dy, dz, w3, h2, Bm, nelv, s, err, skip);
      case 8: {
        const cudaError_t e =
            launch_stress_mma<false>(io, geo, dx, dy, dz, w3, h2, Bm, nelv, s, err, skip);
        if (e != cudaErrorNotSupported) return e;
        break;
      }
      case 10: return launch_stress_tma<10, 2, 5>(io, geo, dx, dy, dz, w3, h2, Bm, nelv, s, err, skip);
      default: break;
    }
  }
  cudaError_t e;
  switch (lx) {
#define NB_STRESS_GEN(L) \
  case L: e = launch_stress_gen<L>(io, geo, dx, dy, dz, w3, nelv, s, skip); break;
    NB_STRESS_GEN(2) NB_STRESS_GEN(3) NB_STRESS_GEN(4) NB_STRESS_GEN(5) NB_STRESS_GEN(6)
    NB_STRESS_GEN(7) NB_STRESS_GEN(8) NB_STRESS_GEN(9) NB_STRESS_GEN(10) NB_STRESS_GEN(11)
    NB_STRESS_GEN(12) NB_STRESS_GEN(13) NB_STRESS_GEN(14) NB_STRESS_GEN(15) NB_STRESS_GEN(16)
#undef NB_STRESS_GEN
    default: return cudaErrorNotSupported;
  }
  if (e != cudaSuccess || !h2) return e;
  return ax_stress_part2(au, av, aw, u, v, w, h2, Bm, (long)nelv * lx * lx * lx, s, skip);
}

// au += h2 B u, av += h2 B v, aw += h2 B w (the reference's part2 kernel,
// ax_helm_full_kernel.h: same products in the same order)
__global__ void ax_stress_part2_kernel(double *__restrict__ au, double *__restrict__ av,
                                       double *__restrict__ aw, const double *__restrict__ u,
                                       const double *__restrict__ v,
                                       const double *__restrict__ w,
                                       const double *__restrict__ h2,
                                       const double *__restrict__ B, long n,
                                       const int *__restrict__ skip) {
  chain();
  if (skip && *skip) return;
  for (long q = blockIdx.x * (long)blockDim.x + threadIdx.x; q < n;
       q += (long)gridDim.x * blockDim.x) {
    au[q] = au[q] + h2[q] * B[q] * u[q];
    av[q] = av[q] + h2[q] * B[q] * v[q];
    aw[q] = aw[q] + h2[q] * B[q] * w[q];
  }
}

cudaError_t ax_stress_part2(double *au, double *av, double *aw, const double *u,
                            const double *v, const double *w, const double *h2,
                            const double *B, long n, cudaStream_t s, const int *skip) {
  if (n <= 0) return cudaSuccess;
  launch_chained(3 * n, ax_stress_part2_kernel, stream_grid(n, 256), 256, 0, s, au, av, aw, u, v,
                 w, h2, B, n,
                                                             skip);
  return cudaGetLastError();
}

// Cofactors and 1/jac of the coordinate map (coef_generate_dxyzdrst,
// src/sem/coef.f90:714-905): the same derivatives and products as the
// geometric factors of the problem.
__global__ void cofactor_kernel(const double *__restrict__ x, const double *__restrict__ y,
                                const double *__restrict__ z, const double *__restrict__ D,
                                int lx, long n, double *__restrict__ cof) {
  extern __shared__ double smc[];
  const int l3 = lx * lx * lx;
  double *sx = smc, *sy = smc + l3, *sz = smc + 2 * l3, *sD = smc + 3 * l3;
  const long e = blockIdx.x;
  for (int q = threadIdx.x; q < l3; q += blockDim.x) {
    sx[q] = x[e * l3 + q];
    sy[q] = y[e * l3 + q];
    sz[q] = z[e * l3 + q];
  }
  for (int q = threadIdx.x; q < lx * lx; q += blockDim.x) sD[q] = D[q];
  __syncthreads();
  for (int p = threadIdx.x; p < l3; p += blockDim.x) {
    const int i = p % lx, j = (p / lx) % lx, k = p / (lx * lx);
    double xr = 0, yr = 0, zr = 0, xs = 0, ys = 0, zs = 0, xt = 0, yt = 0, zt = 0;
    for (int l = 0; l < lx; l++) {
      const double dr = sD[i + lx * l], ds = sD[j + lx * l], dt = sD[k + lx * l];
      const int pr = l + lx * j + lx * lx * k, ps = i + lx * l + lx * lx * k,
                pt = i + lx * j + lx * lx * l;
      xr += dr * sx[pr];
      yr += dr * sy[pr];
      zr += dr * sz[pr];
      xs += ds * sx[ps];
      ys += ds * sy[ps];
      zs += ds * sz[ps];
      xt += dt * sx[pt];
      yt += dt * sy[pt];
      zt += dt * sz[pt];
    }
    double jac = 0.0;
    jac = jac + xr * ys * zt;
    jac = jac + xt * yr * zs;
    jac = jac + xs * yt * zr;
    jac = jac - xr * yt * zs;
    jac = jac - xs * yr * zt;
    jac = jac - xt * ys * zr;
    const long g = e * l3 + p;
    const double v[10] = {ys * zt - yt * zs, xt * zs - xs * zt, xs * yt - xt * ys,
                          yt * zr - yr * zt, xr * zt - xt * zr, xt * yr - xr * yt,
                          yr * zs - ys * zr, xs * zr - xr * zs, xr * ys - xs * yr,
                          1.0 / jac};
    for (int a = 0; a < 10; a++) cof[(size_t)a * n + g] = v[a];
  }
}

}  // namespace nb

using namespace nb;

cudaError_t nb_problem::ensure_cofactors(cudaStream_t s) {
  if (cof) return cudaSuccess;
  double *c = nullptr;
  cudaError_t e = cudaMalloc(&c, (size_t)10 * n * sizeof(double));
  if (e != cudaSuccess) return e;
  const int l3 = lx * lx * lx;
  const size_t sm = (size_t)(3 * l3 + lx * lx) * sizeof(double);
  if (sm > 48 * 1024) {
    e = cudaFuncSetAttribute(cofactor_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sm);
    if (e != cudaSuccess) {
      cudaFree(c);
      return e;
    }
  }
  cofactor_kernel<<<(unsigned)nelv, 256, sm, s>>>(x, y, z, D, lx, n, c);
  e = cudaGetLastError();
  if (e != cudaSuccess) {
    cudaFree(c);
    return e;
  }
  cof = c;
  return cudaSuccess;
}

static void stress_fatal(cudaError_t e, const char *what) {
  if (e == cudaSuccess) return;
  fprintf(stderr, "%s: %s\n", what, cudaGetErrorString(e));
  exit(1);
}

// Part-1 drop-in: cuda_ax_helm_stress_vector
// (src/math/bcknd/device/cuda/ax_helm_full.cu).  Launches on the default
// stream of the drop-ins (Neko's glb_cmd_queue when linked into Neko).
// dxt, dyt, dzt are accepted and unused: the kernels read the transposes out
// of dx, dy, dz, as the reference kernel does.
extern "C" void cuda_ax_helm_stress_vector(void *au, void *av, void *aw, void *u, void *v,
                                           void *w, void *dx, void *dy, void *dz, void *dxt,
                                           void *dyt, void *dzt, void *h1, void *drdx,
                                           void *drdy, void *drdz, void *dsdx, void *dsdy,
                                           void *dsdz, void *dtdx, void *dtdy, void *dtdz,
                                           void *jacinv, void *w3, int *nelv, int *lx) {
  (void)dxt;
  (void)dyt;
  (void)dzt;
  if (*lx < 2 || *lx > 16) {
    fprintf(stderr, "cuda_ax_helm_stress_vector: size not supported: %d\n", *lx);
    exit(1);
  }
  auto d = [](void *p) { return (double *)p; };
  const double *cof[9] = {d(drdx), d(drdy), d(drdz), d(dsdx), d(dsdy),
                          d(dsdz), d(dtdx), d(dtdy), d(dtdz)};
  stress_fatal(ax_stress(d(au), d(av), d(aw), d(u), d(v), d(w), d(dx), d(dy), d(dz), d(h1),
                         d(jacinv), cof, d(w3), *nelv, *lx, default_stream(), nullptr, nullptr,
                         nullptr, nullptr),
               "cuda_ax_helm_stress_vector");
}

extern "C" void cuda_ax_helm_stress_vector_part2(void *au, void *av, void *aw, void *u,
                                                 void *v, void *w, void *h2, void *B, int *n) {
  stress_fatal(ax_stress_part2((double *)au, (double *)av, (double *)aw, (const double *)u,
                               (const double *)v, (const double *)w, (const double *)h2,
                               (const double *)B, *n, default_stream(), nullptr),
               "cuda_ax_helm_stress_vector_part2");
}

namespace nb {
// A_stress (u, v, w) of problem P (with the h2 B term when ifh2) on stream s.
cudaError_t problem_ax_stress(nb_problem *P, double *au, double *av, double *aw,
                              const double *u, const double *v, const double *w,
                              cudaStream_t s, const int *skip) {
  cudaError_t e = P->ensure_cofactors(s);
  if (e != cudaSuccess) return e;
  const long n = P->n;
  const double *cof[9];
  for (int a = 0; a < 9; a++) cof[a] = P->cof + (size_t)a * n;
  // the h2 B term in the same pass where the streaming kernel runs
  return ax_stress(au, av, aw, u, v, w, P->D, P->D, P->D, P->h1, P->cof + (size_t)9 * n, cof,
                   P->w3, P->nelv, P->lx, s, P->err, skip, P->ifh2 ? P->h2 : nullptr,
                   P->ifh2 ? P->B : nullptr);
}
}  // namespace nb

namespace nb {
// The coupled CG's direction update, full-stress operator (with the h2 B
// term) and curvature in one streaming pass (StressCg); returns
// cudaErrorNotSupported where the streaming kernel does not apply.
cudaError_t problem_ax_stress_cg(nb_problem *P, double *const w[3], double *const p[3],
                                 const double *const z[3], CgState *st, double *partials,
                                 unsigned *counter, cudaStream_t s) {
  cudaError_t e = P->ensure_cofactors(s);
  if (e != cudaSuccess) return e;
  const long n = P->n;
  StressIo io{{w[0], w[1], w[2]}, {p[0], p[1], p[2]}};
  StressGeo geo{P->h1, P->cof + (size_t)9 * n, {}};
  for (int a = 0; a < 9; a++) geo.c[a] = P->cof + (size_t)a * n;
  StressCg cg;
  for (int c = 0; c < 3; c++) {
    cg.z[c] = z[c];
    cg.pout[c] = p[c];
  }
  cg.st = st;
  cg.partials = partials;
  cg.counter = counter;
  const void *ptrs[] = {p[0], p[1], p[2], z[0], z[1], z[2], P->h1, P->cof};
  for (const void *q : ptrs)
    if (reinterpret_cast<uintptr_t>(q) & 15) return cudaErrorNotSupported;
  const double *h2 = P->ifh2 ? P->h2 : nullptr, *Bm = P->ifh2 ? P->B : nullptr;
  switch (P->lx) {
    case 4: return launch_stress_tma<4, 2, 4, true>(io, geo, P->D, P->D, P->D, P->w3, h2, Bm, P->nelv, s, P->err, nullptr, cg);
    case 6: return launch_stress_tma<6, 2, 3, true>(io, geo, P->D, P->D, P->D, P->w3, h2, Bm, P->nelv, s, P->err, nullptr, cg);
    case 8: return launch_stress_mma<true>(io, geo, P->D, P->D, P->D, P->w3, h2, Bm, P->nelv, s, P->err, nullptr, cg);
    case 10: return launch_stress_tma<10, 2, 5, true>(io, geo, P->D, P->D, P->D, P->w3, h2, Bm, P->nelv, s, P->err, nullptr, cg);
    default: return cudaErrorNotSupported;
  }
}
}  // namespace nb

extern "C" nb_status nb_ax_stress(nb_problem *p, double *au, double *av, double *aw,
                                  const double *u, const double *v, const double *w,
                                  void *stream) {
  if (!p || !au || !av || !aw || !u || !v || !w) {
    set_error("null argument");
    return NB_ERR_ARG;
  }
  cudaError_t e = problem_ax_stress(p, au, av, aw, u, v, w, (cudaStream_t)stream, nullptr);
  if (e != cudaSuccess) {
    set_error(std::string("nb_ax_stress: ") + cudaGetErrorString(e));
    return e == cudaErrorMemoryAllocation ? NB_ERR_OOM : NB_ERR_CUDA;
  }
  return NB_OK;
}
