// ax_helm.cu -- matrix-free Helmholtz operator w = D^T (h1 G D u) on sm_100a.
//
// The streaming forms, their dispatch and the entry points; other orders and
// unaligned operands take ax_helm_gen.cu and ax_cg_gen.cu.  The FP64 path is
// HBM-bound (72 B and 12 lx + 15 flop per point), so no tensor cores.
//
// Follows the arithmetic of ax_helm_lx (src/math/bcknd/cpu/ax_helm_cpu.f90:
// 180-290): ur = Dx u, us = Dy u, ut = Dz u; (ur,us,ut) <- h1 G (ur,us,ut);
// w = Dxt ur + Dyt us + Dzt ut, with D matrices column-major as passed.
#include <array>
#include <initializer_list>
#include <cstring>
#include <map>
#include <mutex>
#include <vector>
#include <cstdio>
#include <cstdlib>

#include <cstdint>

#include "nb_ax.cuh"
#include "nb_chain.cuh"
#include "nb_kernels.h"
#include "nb_precond.h"
#include "nb_reduce.cuh"
#include "nb_tma.cuh"

namespace nb {

// Error word of the drop-in cuda_ax_helm, which has no problem handle to
// carry one: 0 = ok, 1 = a bulk-copy wait timed out.  The native entry
// points pass their problem's own word instead.  Read and cleared by
// take_dropin_error() (after the synchronising drop-in reductions).
__device__ int nb_dropin_error = 0;

// ---------------------------------------------------------------------------
// Streaming form: a persistent kernel in which each CTA walks its share of the
// elements and keeps S of them in flight in a shared-memory ring.  One thread
// issues, per element, 1-D bulk copies of the arrays it needs (u, h1, G11,
// G22, G33, G12, G13, G23; each lx^3 contiguous values) completing on the
// stage's mbarrier, so the bytes in flight per SM do not depend on register
// pressure.  KS thread groups split the k-planes of an element: thread
// (i, j, kh) computes planes [kh KP, (kh + 1) KP).
//
// A bulk copy moves whole 16-byte units, and lx^3 doubles are none for odd lx:
// those orders stream two elements a stage (NE = 2), which start on a 16-byte
// boundary whenever the array does.  The last element of an odd count arrives
// as lx^3 - 1 copied values and one stored by the issuing thread.  At lx 7 and
// 6.8 M points the general kernel took 181 us (260 with h2), this form takes
// 101 (127): the blocks of the general kernel each wait for their own loads,
// several times an element.
//
// With CG the kernel is fused with the two CG steps around the operator:
// p = z + beta p (cg_update_p), w = A p (element-local, before the
// gather-scatter), and pap = sum over the local points of p * w with alpha =
// rtz / pap (cg_pap).  p is continuous and zero on masked points (z is), so
// the local sum equals (p, mult gs(w)) with the mask, the form the reference
// evaluates after the gather-scatter (cg_device.f90:211-214): each global
// point's weights 1/k over its k copies add up to one.  The ring carries z
// and the old p in place of u; each thread forms the new p for its own
// points, stores it, and the element's operator then reads it from the stage.
//
// The h2 B u term, when h2 is given, is added in the same pass: each thread
// reads h2 and B for its own points, so they cost no shared memory; they are
// brought to L2 when the stage is filled, as their latency is not hidden
// behind the wait otherwise (139 us against the 112 us of 736 MB for a fused
// step on 7.1 M points, now 118).
//
// Bound by HBM: 72 B a point, 88 with the step, 16 more with h2; the next
// limiter is the shared-memory pipe (81 % at lx 8).  At 7.1 M points and lx 8 the
// step takes 105 us, 91 % of the measured copy rate (140 in three launches).
// ---------------------------------------------------------------------------
// AL: the three work planes live in the stage itself, over the G11, G22, G33
// arrays of the element being computed (each thread reads the six factors of a
// point before it writes that point's three fluxes, and no thread reads
// another point's factors), which frees room for a further stage or block; the
// stage is then refilled after the second pass instead of the first.  At lx 8
// the plain operator takes 88.2 us so at 7.1 M points, 90.2 otherwise; at lx 9
// with h2 150 against 166.
template <int LX, int S, int KS, int NE, bool CG, bool AL>
struct AxCfgS {
  static constexpr int L2 = LX * LX, L3 = L2 * LX, NA = CG ? 9 : 8;
  static constexpr int KP = (LX + KS - 1) / KS;
  static constexpr int THREADS = ((L2 * KS * NE + 31) / 32) * 32;
  static constexpr size_t ABYTES = (size_t)L3 * sizeof(double);  // one array of one element
  static constexpr size_t SMEM =
      (S * NA + (AL ? 0 : 3)) * NE * ABYTES + 2 * L2 * sizeof(double) + 16 * S;
  static_assert((NE * L3 * sizeof(double)) % 16 == 0, "stage arrays are whole 16-byte units");
};

template <int LX, int S, int KS, int NE, bool CG, bool AL, bool H2, typename TZ>
__global__ void __launch_bounds__(AxCfgS<LX, S, KS, NE, CG, AL>::THREADS)
    ax_stream_kernel(const AxArgs<TZ> a) {
  using C = AxCfgS<LX, S, KS, NE, CG, AL>;
  constexpr int L2 = C::L2, L3 = C::L3, NA = C::NA, KP = C::KP, THREADS = C::THREADS;
  constexpr int AS = NE * L3;  // one array of a stage
  constexpr int U0 = CG ? 1 : 0;
  static_assert(NE == 1 || !CG || sizeof(TZ) == 8, "FP32 z of odd lx is not a whole unit");
  extern __shared__ __align__(128) unsigned char smem_ring[];
  double *stage = reinterpret_cast<double *>(smem_ring);
  double *sD = stage + (S * NA + (AL ? 0 : 3)) * AS, *sDt = sD + L2;
  uint64_t *full = reinterpret_cast<uint64_t *>(sDt + L2);

  const int tid = threadIdx.x;
  const int G = gridDim.x, b = blockIdx.x;
  const int ngroup = (a.nelv + NE - 1) / NE;
  const int nt = b < ngroup ? (ngroup - b + G - 1) / G : 0;
  if (tid == 0) {
    for (int s = 0; s < S; s++) mbar_init(&full[s], 1);
    fence_barrier_init();
  }
  chain();
  if (a.skip && *a.skip) return;
  if (CG && a.st && a.st->done) return;
  const double beta = CG ? (a.st ? a.st->beta : a.beta) : 0.0;
  for (int q = tid; q < L2; q += THREADS) {
    sD[q] = a.D[q];
    sDt[q] = a.Dt[q];
  }
  __syncthreads();
  // stage arrays: (z, p) or u, h1, G11, G22, G33, G12, G13, G23
  auto issue = [&](int t, int s) {
    const long e0 = ((long)b + (long)t * G) * NE;
    const bool odd = NE == 2 && e0 + 1 == a.nelv;  // the last element alone
    const uint32_t count = (uint32_t)(odd ? L3 - 1 : AS);  // values an array copies
    double *base = stage + (size_t)s * NA * AS;
    auto source = [&](int q) {
      return q < U0 ? nullptr
                    : q == U0 ? (CG ? (const double *)a.p : a.u)
                              : q == U0 + 1 ? a.h1 : a.g[q - U0 - 2];
    };
    if (odd) {  // its last value of each array, before the arrival below
      if (CG) reinterpret_cast<TZ *>(base)[L3 - 1] = a.z[e0 * L3 + L3 - 1];
#pragma unroll
      for (int q = U0; q < NA; q++) base[(size_t)q * AS + L3 - 1] = source(q)[e0 * L3 + L3 - 1];
    }
    const uint32_t zbytes = CG ? count * (uint32_t)sizeof(TZ) : 0u;
    mbar_arrive_expect_tx(&full[s], (uint32_t)(NA - U0) * count * 8u + zbytes);
    if (CG) bulk_g2s(base, a.z + e0 * L3, zbytes, &full[s]);
#pragma unroll
    for (int q = U0; q < NA; q++)
      bulk_g2s(base + (size_t)q * AS, source(q) + e0 * L3, count * 8u, &full[s]);
    if (H2) {
      bulk_prefetch_l2(a.h2 + e0 * L3, count * 8u);
      bulk_prefetch_l2(a.B + e0 * L3, count * 8u);
    }
  };
  if (tid == 0)
    for (int t = 0; t < S && t < nt; t++) issue(t, t);

  const int col = tid % L2, part = tid / L2;
  const int kh = NE == 1 ? part : part % KS, el = NE == 1 ? 0 : part / KS;
  const int i = col % LX, j = col / LX, k0 = kh * KP;
  double Di[LX], Dj[LX], Dti[LX], Dtj[LX];
#pragma unroll
  for (int l = 0; l < LX; l++) {
    Di[l] = sD[i + LX * l];
    Dj[l] = sD[j + LX * l];
    Dti[l] = sDt[i + LX * l];
    Dtj[l] = sDt[j + LX * l];
  }

  double pap = 0.0;
  int t = 0;
  bool failed = false;
  for (; t < nt; t++) {
    const int s = t % S;
    const long e = ((long)b + (long)t * G) * NE + el;
    const bool act = (L2 * KS * NE == THREADS || tid < L2 * KS * NE) && (NE == 1 || e < a.nelv);
    auto plane = [&](int kk) { return LX % KS == 0 || k0 + kk < LX; };
    const bool ok = mbar_wait(&full[s], (uint32_t)((t / S) & 1));
    if (__syncthreads_or(!ok)) {
      failed = true;
      break;
    }
    double *base = stage + (size_t)s * NA * AS;
    double *su = base + U0 * AS + el * L3;  // u, or the old p replaced by the new
    const double *sh = su + AS, *s11 = su + 2 * AS, *s22 = su + 3 * AS, *s33 = su + 4 * AS,
                 *s12 = su + 5 * AS, *s13 = su + 6 * AS, *s23 = su + 7 * AS;
    // work planes: separate, or over this stage's G11, G22, G33 (AL)
    double *wr = AL ? su + 2 * AS : stage + (size_t)S * NA * AS + el * L3, *ws = wr + AS,
           *wt = ws + AS;
    if constexpr (CG) {
      const TZ *sz = reinterpret_cast<const TZ *>(base) + el * L3;
      if (act) {
#pragma unroll
        for (int kk = 0; kk < KP; kk++)
          if (plane(kk)) {
            const int q = col + L2 * (k0 + kk);
            const double pn = (double)sz[q] + beta * su[q];
            su[q] = pn;
            a.p[e * L3 + q] = pn;
          }
      }
      __syncthreads();  // the new p complete in the stage
    }
    double own[H2 || CG ? KP : 1];  // u (p) at this thread's points
    if (act) {
      double ru[LX];  // its column
#pragma unroll
      for (int l = 0; l < LX; l++) ru[l] = su[col + L2 * l];
      if constexpr (H2 || CG) {
#pragma unroll
        for (int kk = 0; kk < KP; kk++)
          if (plane(kk)) own[kk] = su[col + L2 * (k0 + kk)];
      }
#pragma unroll
      for (int kk = 0; kk < KP; kk++) {
        if (!plane(kk)) continue;
        const int k = k0 + kk;
        double ur = 0, us = 0, ut = 0;
#pragma unroll
        for (int l = 0; l < LX; l++) {
          ur += Di[l] * su[l + LX * j + L2 * k];
          us += Dj[l] * su[i + LX * l + L2 * k];
          ut += sD[k + LX * l] * ru[l];
        }
        const int q = col + L2 * k;
        const double H = sh[q];
        const double a11 = s11[q], a22 = s22[q], a33 = s33[q], a12 = s12[q], a13 = s13[q],
                     a23 = s23[q];
        wr[q] = H * (a11 * ur + a12 * us + a13 * ut);
        ws[q] = H * (a12 * ur + a22 * us + a23 * ut);
        wt[q] = H * (a13 * ur + a23 * us + a33 * ut);
      }
    }
    // AL: this thread's writes over the factors come before the next copy
    if (AL || CG) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();  // stage s consumed (but for AL's planes), work planes complete
    if (!AL && tid == 0 && t + S < nt) issue(t + S, s);
    if (act) {
      double h2v[H2 ? KP : 1], bv[H2 ? KP : 1];  // in flight during the contractions
      if constexpr (H2) {
#pragma unroll
        for (int kk = 0; kk < KP; kk++)
          if (plane(kk)) {
            const long g = e * L3 + col + L2 * (k0 + kk);
            h2v[kk] = __ldg(a.h2 + g);
            bv[kk] = __ldg(a.B + g);
          }
      }
      double rt[LX];
#pragma unroll
      for (int l = 0; l < LX; l++) rt[l] = wt[col + L2 * l];
#pragma unroll
      for (int kk = 0; kk < KP; kk++) {
        if (!plane(kk)) continue;
        const int k = k0 + kk;
        double x = 0, y = 0, z = 0;
#pragma unroll
        for (int l = 0; l < LX; l++) {
          x += Dti[l] * wr[l + LX * j + L2 * k];
          y += Dtj[l] * ws[i + LX * l + L2 * k];
          z += sDt[k + LX * l] * rt[l];
        }
        double wq = x + y + z;
        if constexpr (H2) wq = wq + h2v[kk] * bv[kk] * own[kk];
        a.w[e * L3 + col + L2 * k] = wq;
        if constexpr (CG) pap += own[kk] * wq;
      }
    }
    __syncthreads();  // work planes free for the next element
    if (AL && tid == 0 && t + S < nt) issue(t + S, s);
  }
  if (failed) {
    if (tid == 0) {
      atomicExch(a.err ? a.err : &nb_dropin_error, 1);
      // bounded wait for this CTA's copies still in flight
      for (int q = t; q < nt && q < t + S; q++) mbar_wait(&full[q % S], (uint32_t)((q / S) & 1));
    }
    __syncthreads();
  }
  if constexpr (CG) {
    double tot;  // every block takes part, a failed one with its partial sum
    if (grid_sum<THREADS>(pap, a.partials, a.counter, &tot)) {
      if (a.st) {
        a.st->pap = tot;
        a.st->alpha = a.st->rtz1 / tot;
      } else if (a.pap_out) {
        *a.pap_out = tot;
      }
    }
  }
}

template <int LX, int S, int KS, int NE, bool CG, bool AL, bool H2, typename TZ>
static cudaError_t launch_ax_stream_as(const AxArgs<TZ> &a, cudaStream_t st) {
  using C = AxCfgS<LX, S, KS, NE, CG, AL>;
  auto kern = ax_stream_kernel<LX, S, KS, NE, CG, AL, H2, TZ>;
  static int grid_per_dev[64] = {0};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  int &g = grid_per_dev[dev & 63];
  if (g == 0) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
    if (e != cudaSuccess) return e;
    int per_sm = 0, sms = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, C::THREADS, C::SMEM);
    if (e != cudaSuccess) return e;
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    g = (per_sm > 0 ? per_sm : 1) * sms;
  }
  if (a.nelv <= 0) return cudaSuccess;
  const int ngroup = (a.nelv + NE - 1) / NE;
  int grid = ngroup < g ? ngroup : g;
  if (CG && grid > a.max_grid) grid = a.max_grid;
  return launch_chained((long)a.nelv * C::L3, kern, grid, C::THREADS, C::SMEM, st, a);
}

// Stages, k split and overlay of an order, without and with h2.  A larger split
// (more threads an element) hides the loads of h2 and B, which come past the
// ring: lx 8 with h2 takes 102 us at 7.1 M points split by 4, 126 by 2.  A
// smaller one loads less from shared memory, as every part of the split reads
// its columns whole for the t derivatives: the step at lx 8 takes 105 us at 7.1
// M points unsplit, 113 split by 2; at lx 10 128 us at 6.9 M points split by 2,
// 156 by 5 (with a third, overlaid stage).
template <int LX, int NE, bool CG, int S, int KS, bool AL, int S2, int KS2, bool AL2, typename TZ>
static cudaError_t launch_ax_stream(const AxArgs<TZ> &a, cudaStream_t st) {
  return a.h2 ? launch_ax_stream_as<LX, S2, KS2, NE, CG, AL2, true>(a, st)
              : launch_ax_stream_as<LX, S, KS, NE, CG, AL, false>(a, st);
}

// Whether the streaming form takes the operands: every copied array on a
// 16-byte boundary.
static bool bulk_aligned(std::initializer_list<const void *> ptrs) {
  for (const void *p : ptrs)
    if (reinterpret_cast<uintptr_t>(p) & 15) return false;
  return true;
}

// Dispatch of the streaming operator; returns cudaErrorNotSupported when no
// instantiation covers lx or a pointer is not 16-byte aligned.
cudaError_t ax_helm_stream(double *w, const double *u, const double *D, const double *Dt,
                           const double *h1, const double *g11, const double *g22,
                           const double *g33, const double *g12, const double *g13,
                           const double *g23, const double *h2, const double *B, int nelv, int lx,
                           cudaStream_t s, const int *skip, int *err) {
  if (!bulk_aligned({u, h1, g11, g22, g33, g12, g13, g23, h2, B})) return cudaErrorNotSupported;
  AxArgs<double> a{};
  a.w = w, a.u = u, a.D = D, a.Dt = Dt, a.h1 = h1;
  a.g[0] = g11, a.g[1] = g22, a.g[2] = g33, a.g[3] = g12, a.g[4] = g13, a.g[5] = g23;
  a.h2 = h2, a.B = B, a.nelv = nelv, a.skip = skip, a.err = err;
  switch (lx) {
    case 4: return launch_ax_stream<4, 1, false, 4, 4, false, 4, 4, false>(a, s);
    case 5: return launch_ax_stream<5, 2, false, 3, 1, false, 3, 1, false>(a, s);
    case 6: return launch_ax_stream<6, 1, false, 3, 3, false, 3, 3, false>(a, s);
    case 7:
      // While a block (two a multiprocessor) takes three pairs of elements at
      // most, a single stage: the copies of a second would share the bandwidth
      // with those of the first pair, which every block waits for.  Out of cache,
      // operator with h2 and gather-scatter: 26 us against 30 with two stages on
      // 1320 elements, 30 and 34 on 1760, 44 and 46 on 3000, 52 and 52 on 4000, 73
      // and 62 on 6000; in cache the operator alone takes 12.3 and 11.6 us on 1320,
      // 27.7 and 23.5 on 3000.
      return nelv <= 12 * device_sms()
                 ? launch_ax_stream<7, 2, false, 1, 2, false, 1, 2, false>(a, s)
                 : launch_ax_stream<7, 2, false, 2, 1, false, 2, 2, false>(a, s);
    case 8: return launch_ax_stream<8, 1, false, 2, 2, true, 2, 4, false>(a, s);
    case 9: return launch_ax_stream<9, 2, false, 1, 3, false, 2, 2, true>(a, s);
    case 10: return launch_ax_stream<10, 1, false, 2, 5, false, 2, 2, false>(a, s);
    default: return cudaErrorNotSupported;
  }
}

template <typename TZ>
cudaError_t ax_cg_fused(double *w, double *p, const TZ *z, const double *D, const double *Dt,
                        const double *h1, const double *g11, const double *g22, const double *g33,
                        const double *g12, const double *g13, const double *g23,
                        const double *h2, const double *B, int nelv, int lx, CgState *st,
                        double beta, double *pap_out, double *partials, unsigned *counter,
                        int max_grid, cudaStream_t s, int *err) {
  if (nelv <= 0) return cudaErrorNotSupported;
  AxArgs<TZ> a{};
  a.w = w, a.p = p, a.z = z, a.D = D, a.Dt = Dt, a.h1 = h1;
  a.g[0] = g11, a.g[1] = g22, a.g[2] = g33, a.g[3] = g12, a.g[4] = g13, a.g[5] = g23;
  a.h2 = h2, a.B = B, a.nelv = nelv, a.err = err;
  a.st = st, a.beta = beta, a.pap_out = pap_out, a.partials = partials, a.counter = counter;
  a.max_grid = max_grid;
  const bool rest = bulk_aligned({p, h1, g11, g22, g33, g12, g13, g23, h2, B});
  // z alone off a 16-byte boundary: beyond 2^20 points the separate passes, whose
  // operator streams p, are faster than the general kernel at these orders (lx 10,
  // 2.7 M points: 72 us, 90; lx 8 58 and 62), below it is the launches that count
  // (lx 8, 369 thousand points: 23 us, 13)
  if (rest && !bulk_aligned({z}) && (lx == 6 || lx == 8 || lx == 10) &&
      (long)nelv * lx * lx * lx > (1L << 20))
    return cudaErrorNotSupported;
  if (rest && bulk_aligned({z})) {
    switch (lx) {
      case 4: return launch_ax_stream<4, 1, true, 4, 4, false, 4, 4, false>(a, s);
      case 6: return launch_ax_stream<6, 1, true, 3, 3, false, 3, 3, false>(a, s);
      case 8: return launch_ax_stream<8, 1, true, 2, 1, false, 2, 2, false>(a, s);
      case 10: return launch_ax_stream<10, 1, true, 2, 2, false, 2, 2, false>(a, s);
      default: break;
    }
    if constexpr (sizeof(TZ) == 8) {  // pairs of FP32 z are not whole 16-byte units
      switch (lx) {
        case 5: return launch_ax_stream<5, 2, true, 2, 2, false, 2, 2, false>(a, s);
        case 7: return launch_ax_stream<7, 2, true, 1, 2, false, 1, 2, false>(a, s);
        case 9: return launch_ax_stream<9, 2, true, 1, 3, false, 2, 2, true>(a, s);
        default: break;
      }
    }
  }
  return ax_cg_general<TZ>(a, lx, s);
}
template cudaError_t ax_cg_fused<double>(double *, double *, const double *, const double *,
                                         const double *, const double *, const double *,
                                         const double *, const double *, const double *,
                                         const double *, const double *, const double *,
                                         const double *, int, int, CgState *, double, double *,
                                         double *, unsigned *, int, cudaStream_t, int *);
template cudaError_t ax_cg_fused<float>(double *, double *, const float *, const double *,
                                        const double *, const double *, const double *,
                                        const double *, const double *, const double *,
                                        const double *, const double *, const double *,
                                        const double *, int, int, CgState *, double, double *,
                                        double *, unsigned *, int, cudaStream_t, int *);

int *dropin_error_word() {
  static int *cache[64] = {nullptr};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  if (!cache[dev]) {
    void *p = nullptr;
    if (cudaGetSymbolAddress(&p, nb_dropin_error) != cudaSuccess) return nullptr;
    cache[dev] = (int *)p;
  }
  return cache[dev];
}

int take_dropin_error() {
  int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, nb_dropin_error, sizeof(int)) != cudaSuccess) return -1;
  if (v) cudaMemcpyToSymbol(nb_dropin_error, &zero, sizeof(int));
  return v;
}

}  // namespace nb

namespace nb {
// Whether a space's dx, dy, dz (and dxt, dyt, dzt) hold the same matrix.
// Neko keeps them as three device arrays with equal contents for GLL
// spaces; the streaming kernel needs one matrix, so the contents are
// compared once per set of pointers (after the default stream has drained)
// and the answer is kept.
bool same_derivatives(const void *dx, const void *dy, const void *dz, const void *dxt,
                      const void *dyt, const void *dzt, int lx) {
  if (dx == dy && dx == dz && dxt == dyt && dxt == dzt) return true;
  static std::mutex mu;
  static std::map<std::array<const void *, 6>, std::pair<int, bool>> known;
  const std::array<const void *, 6> key{dx, dy, dz, dxt, dyt, dzt};
  std::lock_guard<std::mutex> lock(mu);
  auto it = known.find(key);
  if (it != known.end() && it->second.first == lx) return it->second.second;
  bool same = false;
  if (cudaStreamSynchronize(default_stream()) == cudaSuccess) {
    const size_t b = (size_t)lx * lx * sizeof(double);
    std::vector<char> m[6];
    bool ok = true;
    for (int q = 0; q < 6 && ok; q++) {
      m[q].resize(b);
      ok = cudaMemcpy(m[q].data(), key[q], b, cudaMemcpyDeviceToHost) == cudaSuccess;
    }
    same = ok && !memcmp(m[0].data(), m[1].data(), b) && !memcmp(m[0].data(), m[2].data(), b) &&
           !memcmp(m[3].data(), m[4].data(), b) && !memcmp(m[3].data(), m[5].data(), b);
  }
  known[key] = {lx, same};
  return same;
}
}  // namespace nb

extern "C" void cuda_ax_helm(void *w, void *u, void *dx, void *dy, void *dz, void *dxt,
                             void *dyt, void *dzt, void *h1, void *g11, void *g22, void *g33,
                             void *g12, void *g13, void *g23, int *nelv, int *lx) {
  if (*lx < 2 || *lx > 16) {
    fprintf(stderr, "cuda_ax_helm: unsupported lx %d (2..16)\n", *lx);
    exit(1);
  }
  cudaError_t e = cudaErrorNotSupported;
  if (nb::same_derivatives(dx, dy, dz, dxt, dyt, dzt, *lx))
    e = nb::ax_helm_stream((double *)w, (const double *)u, (const double *)dx,
                                   (const double *)dxt, (const double *)h1, (const double *)g11,
                                   (const double *)g22, (const double *)g33, (const double *)g12,
                                   (const double *)g13, (const double *)g23, nullptr, nullptr,
                                   *nelv, *lx, nb::default_stream(), nullptr, nullptr);
  if (e == cudaErrorNotSupported)
    e = nb::ax_helm<double>(
      (double *)w, (const double *)u, (const double *)dx, (const double *)dy,
      (const double *)dz, (const double *)dxt, (const double *)dyt, (const double *)dzt,
      (const double *)h1, (const double *)g11, (const double *)g22, (const double *)g33,
      (const double *)g12, (const double *)g13, (const double *)g23, *nelv, *lx,
      nb::default_stream(), nullptr);
  nb::cuda_check_fatal(e, "cuda_ax_helm");
}
