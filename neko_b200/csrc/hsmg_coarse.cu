// hsmg_coarse.cu -- the coarse end of hsmg.
//
// The reference runs the coarse level of pc_hsmg (src/krylov/pc_hsmg.f90:
// 540-560) as separate steps: restrict the middle-level residual (times
// mult) to lx = 2, gather-scatter and mask it, run `niter` Jacobi-CG
// iterations (cg.f90, each with its own vector kernels, Ax, gs and three
// reductions), then prolong the correction back to the middle level.  On the
// vertices every one of those steps is a fraction of a microsecond of work,
// so what it costs is the latency of the steps between its reductions.
//
// Here the coarse problem lives on its distinct unmasked vertices as a
// sparse matrix (nb_nodes.h): the gather-scatter is gone, vectors are eight
// times shorter, and an iteration is
//
//   p = z + beta p | w = A p, (p, w) | x += alpha p, r -= alpha w, z = d r,
//                                      (r, r), (r, z) |
//
// between barriers (|).  The whole solve is one thread-block cluster (up to
// 16 blocks on one GPC): its barriers are hardware barriers, and its sums
// travel through distributed shared memory, every warp's partial straight to
// every block.  The vectors of a row stay in the registers of the thread that
// owns it, the matrix in the shared memory of its block when it fits, and each
// block holds all of z and p in shared memory: a thread sends its z to every
// block before the barrier of the sums, and each block forms p for itself,
// which leaves two cluster barriers an iteration and gathers that never leave
// the block.  That takes one row a thread, 8192 vertices; larger meshes, and
// those without a mask beyond kCoarseFreeNodes, keep element-local vectors on a
// grid of all multiprocessors (coarse_cg_grid_kernel).
//
// A solve on 343 vertices (8^3 elements) took 124 us as a cooperative grid
// with barriers in global memory and element-local vectors (33 barriers of
// about 3.7 us with their sums), 67 us as a cluster with p in global memory
// and 33 us so.  A cluster leaves the other multiprocessors to the fine-level
// smoother, which runs beside it; the grid form holds one block on every one.
//
// The arithmetic is that of cg_init / cg_precond_dot / cg_update_p /
// ax_helm / gs / cg_update_xr with sums over distinct points: a mult-weighted
// sum over the copies of a point is one term here, and (p, w) of the
// assembled operator is the reference's (p, mult gs(w)).
#include <cmath>
#include <string>

#include "nb_chain.cuh"
#include "nb_cluster.cuh"
#include "nb_gs_dev.cuh"
#include "nb_nodes.h"
#include "nb_precond.h"
#include "nb_reduce.cuh"
#include "nb_tma.cuh"

namespace nb {

// rows a block aims at when the cluster grows: below, the block's own work is
// shorter than a larger cluster's barrier (an hsmg application at lx 8 with 64, 128,
// 256 and 512 rows: 75, 72, 71 and 71 us on 8^3 elements, 90, 82, 82 and 82 on 10^3,
// 97, 97, 93 and 88 on 12^3, 150, 149, 149 and 147 on 16^3)
constexpr int kCoarseRowsPerBlock = 128;
// shared memory a block may spend on its part of the matrix and the vectors
constexpr size_t kCoarseStageBytes = 200 * 1024;
static_assert(kMaxCluster * kCoarseThreads * 2 * sizeof(double) <= kCoarseStageBytes,
              "z and p of the resident form fit");

// f(o,p,r) = sum_k J(k,r) sum_j J(j,p) sum_i J(i,o) (w mult)(i,j,k) per
// element, in T and in the order of tensor3_kernel (x, then y, then z); one
// thread a vertex of an element, 32 elements a block.
template <typename T, int LM>
__global__ void __launch_bounds__(256)
    coarse_restrict_kernel(const T *__restrict__ w_mid, const T *__restrict__ mult_m,
                           const T *__restrict__ J, double *__restrict__ f, long nc,
                           const int *__restrict__ skip) {
  chain();
  if (skip && *skip) return;
  constexpr int M3 = LM * LM * LM;
  constexpr int NE = 32;  // elements a block: its products read once, coalesced
  __shared__ T sJ[LM * 2];  // J(m, c) at m + LM c
  __shared__ T sw[NE * M3 + NE];  // pitch M3 + 1
  const int tid = threadIdx.x;
  if (tid < LM * 2) sJ[tid] = J[tid];
  const long e0 = (long)blockIdx.x * NE;
  {
    const long base = e0 * M3, left = (nc >> 3) * M3 - base;
    constexpr int R = NE * M3 / 256 + (NE * M3 % 256 != 0);
    T a[R], b[R];
#pragma unroll
    for (int g = 0; g < R; g++) {
      const int q = tid + 256 * g;
      const bool ok = q < NE * M3 && q < left;
      a[g] = ok ? __ldg(w_mid + base + q) : T(0);
      b[g] = ok ? __ldg(mult_m + base + q) : T(0);
    }
#pragma unroll
    for (int g = 0; g < R; g++) {
      const int q = tid + 256 * g;
      if (q < NE * M3) sw[q + q / M3] = a[g] * b[g];
    }
  }
  __syncthreads();
  const long q = blockIdx.x * 256L + tid;
  if (q >= nc) return;
  const int o = q & 1, pp = (q >> 1) & 1, rr = (q >> 2) & 1;
  const T *in = sw + (tid >> 3) * (M3 + 1);
  T acc_z = 0;
#pragma unroll
  for (int k = 0; k < LM; k++) {
    T acc_y = 0;
#pragma unroll
    for (int j = 0; j < LM; j++) {
      T acc_x = 0;
#pragma unroll
      for (int i = 0; i < LM; i++) acc_x += sJ[i + LM * o] * in[i + LM * (j + LM * k)];
      acc_y += sJ[j + LM * pp] * acc_x;
    }
    acc_z += sJ[k + LM * rr] * acc_y;
  }
  f[q] = (double)acc_z;
}

// sum of the element-local right-hand side over a node's copies, in order
__device__ __forceinline__ double node_rhs(const NodeOp &A, const double *__restrict__ f,
                                           int row) {
  const int k0 = __ldg(A.eptr + row), k1 = __ldg(A.eptr + row + 1);
  double acc = 0.0;
  for (int k = k0; k < k1; k += 8) {  // eight copies at a time, loads in flight together
    int q[8];
    double v[8];
#pragma unroll
    for (int u = 0; u < 8; u++) q[u] = k + u < k1 ? __ldg(A.ent + k + u) : -1;
#pragma unroll
    for (int u = 0; u < 8; u++) v[u] = q[u] >= 0 ? f[q[u]] : 0.0;
#pragma unroll
    for (int u = 0; u < 8; u++) acc += v[u];
  }
  return acc;
}

// The solve with at most one row a thread: all of z and p in every block's
// shared memory.
__global__ void __launch_bounds__(kCoarseThreads) coarse_cg_resident_kernel(const CoarseCg a) {
  chain();
  if (a.skip && *a.skip) return;
  extern __shared__ __align__(16) unsigned char coarse_smem[];
  __shared__ ClusterSums sums;
  const NodeOp &A = a.A;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const unsigned rank = cluster_rank(), nblk = gridDim.x;
  const int s = wid * (int)nblk + (int)rank, row = 32 * s + lane;
  const bool own = s < A.ns && row < A.nn;
  double *zf = reinterpret_cast<double *>(coarse_smem), *pf = zf + A.nn;
  double *sval = pf + A.nn;
  int *scol = reinterpret_cast<int *>(sval + (size_t)a.stage_slices * A.maxw * 32);
  const double *val = nullptr;
  const int *col = nullptr;
  int width = 0;
  if (s < A.ns) {
    const int o = __ldg(A.soff + s);
    width = __ldg(A.soff + s + 1) - o;
    val = A.val + 32 * (size_t)o + lane;
    col = A.col + 32 * (size_t)o + lane;
    if (a.stage_slices > 0) {
      const size_t to = (size_t)wid * A.maxw * 32;
      stage_slice(A, s, sval + to, scol + to, lane);
      val = sval + to + lane;
      col = scol + to + lane;
    }
  }
  for (int i = tid; i < A.nn; i += kCoarseThreads) pf[i] = 0.0;
  double x = 0.0, r = own ? node_rhs(A, a.f, row) : 0.0;
  const double d = own ? __ldg(A.dinv + row) : 0.0;
  double z = d * r;
  cluster_barrier();  // every block runs before its shared memory is written to
  auto send_z = [&] {
    if (own)
      for (unsigned b = 0; b < nblk; b++) cluster_store(zf + row, b, z);
  };
  send_z();
  double rtr, rtz;
  cluster_allsum2(r * r, r * z, sums, 0, rank, nblk, rtr, rtz);
  double rn = sqrt(rtr) * a.norm_fac;
  bool done = fabs(rn) < 2.220446049250313e-16;
  int iter = 0;
  double rtz_old = 1.0;
  while (!done) {
    const double beta = iter == 0 ? 0.0 : rtz / rtz_old;
    for (int i = tid; i < A.nn; i += kCoarseThreads) pf[i] = zf[i] + beta * pf[i];
    __syncthreads();
    double w = 0.0, p = 0.0;
    if (own) {
      w = row_dot(val, col, width, [&](int c) { return pf[c]; });
      p = pf[row];
    }
    double pap, unused;
    cluster_allsum2(p * w, 0.0, sums, 1, rank, nblk, pap, unused);
    const double alpha = rtz / pap, malpha = -alpha;
    x = x + alpha * p;
    r = r + malpha * w;
    z = d * r;
    if (!own) r = z = 0.0;  // a NaN alpha stays with the rows
    send_z();
    double rtz_new;
    cluster_allsum2(r * r, r * z, sums, 0, rank, nblk, rtr, rtz_new);
    rtz_old = rtz;
    rtz = rtz_new;
    rn = sqrt(rtr) * a.norm_fac;
    iter += 1;
    done = !(rn == rn) || isinf(rn) || rn < a.tol || iter >= a.niter;
  }
  if (own) a.x[row] = x;
}

// ---------------------------------------------------------------------------
// The solve on more vertices: element-local vectors (eight values an element),
// operator and gather-scatter as phases of one cooperative launch, separated by
// grid barriers:
//
//   gs + mask (f) -> | x, p = 0, r = f, z = d r, (r,r), (r,z) -> |
//   per iteration: p = z + beta p, w = A p (element-local), (p, w) -> |
//                  gs + mask (w) -> | x += alpha p, r -= alpha w, z = d r,
//                  (r, r), (r, z) -> |
//
// A flexible CG on a large mesh without a mask amplifies a change of rounding
// in its preconditioner many times over (kCoarseFreeNodes), so this form keeps
// the order of its sums, block by block, at every size.
//
// With at most kU points a thread, x, r, z and p of a point stay in the
// registers of the thread that owns it (20 vector passes an iteration through
// L2 become 11: 116 us a solve on 262144 points, 162 with all of them); only w,
// which the gather-scatter reads across threads, and the solution go to memory.
// 64 registers a thread leave room for other blocks beside this one and take
// 132 us; a cluster of 16 blocks taking the grid's blocks in turn takes 590.
//
// Barriers are bounded: a block that polls too long sets the error word and
// returns; the others then time out at the same barrier and return too.
// ---------------------------------------------------------------------------
constexpr int kU = 4;   // points per thread whose loads are issued together
constexpr int kUA = 2;  // the same for the operator phase (seven operands a point)
constexpr unsigned kBarrierPolls = 1u << 22;

// Grid barrier on one 32-bit word: every block adds 1 except block 0,
// which adds 2^31 - (blocks - 1), so the word's top bit flips exactly when
// the last block arrives (the arrive pattern of cooperative grid sync).
// Arrival is a release and the poll an acquire at gpu scope, so the writes
// of every block before the barrier are visible to every block after it.
__device__ __forceinline__ bool grid_barrier(unsigned *bar, int *err,
                                             unsigned max_polls = kBarrierPolls) {
  __shared__ int ok_s;
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1;
    const unsigned add = blockIdx.x == 0 ? 0x80000000u - (gridDim.x - 1) : 1u;
    unsigned old, v;
    asm volatile("atom.add.release.gpu.u32 %0, [%1], %2;" : "=r"(old) : "l"(bar), "r"(add)
                 : "memory");
    unsigned polls = 0;
    for (;;) {
      asm volatile("ld.acquire.gpu.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
      if ((old ^ v) & 0x80000000u) break;
      if (++polls > max_polls || *(volatile int *)err) {
        ok = 0;
        break;
      }
    }
    if (!ok) atomicExch(err, 1);
    ok_s = ok;
  }
  __syncthreads();
  return ok_s != 0;
}

// Two sums over the grid, identical in every block: each block writes its
// partials, passes the barrier and adds all of them in block order.  buf holds
// 2 * gridDim doubles; consecutive calls must alternate buffers.
__device__ __forceinline__ bool grid_allsum2(double v0, double v1, double *buf, unsigned *bar,
                                             int *err, double &t0, double &t1) {
  __shared__ double sh[2][kCoarseThreads / 32];
  __shared__ double res[2];
  block_sum2<kCoarseThreads>(v0, v1, sh);
  if (threadIdx.x == 0) {
    buf[2 * blockIdx.x] = v0;
    buf[2 * blockIdx.x + 1] = v1;
  }
  if (!grid_barrier(bar, err)) return false;
  double s0 = 0.0, s1 = 0.0;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += kCoarseThreads) {
    s0 += __ldcg(buf + 2 * b);
    s1 += __ldcg(buf + 2 * b + 1);
  }
  block_sum2<kCoarseThreads>(s0, s1, sh);
  if (threadIdx.x == 0) {
    res[0] = s0;
    res[1] = s1;
  }
  __syncthreads();
  t0 = res[0];
  t1 = res[1];
  return true;
}

// w = A p on one lx = 2 element held by 8 consecutive lanes (lane & 7 is the
// point (i, j, k) = (bit0, bit1, bit2)); the arithmetic of ax_helm_kernel.
__device__ __forceinline__ double ax_lx2(double p, int lane, const double *D, const double *Dt,
                                         double H, double G11, double G22, double G33, double G12,
                                         double G13, double G23) {
  const unsigned full = 0xffffffffu;
  const int b = lane & ~7, q = lane & 7, i = q & 1, j = (q >> 1) & 1, k = q >> 2;
  const double ux0 = __shfl_sync(full, p, b + 0 + 2 * j + 4 * k);
  const double ux1 = __shfl_sync(full, p, b + 1 + 2 * j + 4 * k);
  const double uy0 = __shfl_sync(full, p, b + i + 0 + 4 * k);
  const double uy1 = __shfl_sync(full, p, b + i + 2 + 4 * k);
  const double uz0 = __shfl_sync(full, p, b + i + 2 * j + 0);
  const double uz1 = __shfl_sync(full, p, b + i + 2 * j + 4);
  double ur = 0, us = 0, ut = 0;
  ur += D[i] * ux0;
  ur += D[i + 2] * ux1;
  us += D[j] * uy0;
  us += D[j + 2] * uy1;
  ut += D[k] * uz0;
  ut += D[k + 2] * uz1;
  const double a = H * (G11 * ur + G12 * us + G13 * ut);
  const double c = H * (G12 * ur + G22 * us + G23 * ut);
  const double d = H * (G13 * ur + G23 * us + G33 * ut);
  const double a0 = __shfl_sync(full, a, b + 0 + 2 * j + 4 * k);
  const double a1 = __shfl_sync(full, a, b + 1 + 2 * j + 4 * k);
  const double c0 = __shfl_sync(full, c, b + i + 0 + 4 * k);
  const double c1 = __shfl_sync(full, c, b + i + 2 + 4 * k);
  const double d0 = __shfl_sync(full, d, b + i + 2 * j + 0);
  const double d1 = __shfl_sync(full, d, b + i + 2 * j + 4);
  double acc = 0, acc2 = 0, acc3 = 0;
  acc += Dt[i] * a0;
  acc += Dt[i + 2] * a1;
  acc2 += Dt[j] * c0;
  acc2 += Dt[j + 2] * c1;
  acc3 += Dt[k] * d0;
  acc3 += Dt[k + 2] * d1;
  return acc + acc2 + acc3;
}

// The thread's first gather-scatter item, its point indices kept in shared
// memory for the whole launch (the coarse solve runs the same gather-scatter
// eleven times): kind 0 none, 1 pair, 2 segment of up to kGsCache points,
// 3 masked point, 4 not cached (longer segment: gs_add_item each time).
constexpr int kGsCache = 8;
struct GsSlot {
  int idx[kGsCache];
  int kind, len, masked;
};

__device__ __forceinline__ void gs_cache_item(GsSlot &c, const GsDevice &g, long t) {
  c.kind = 0;
  if (t >= gs_items(g, true)) return;
  if (t < g.npairs) {
    const int2 p = __ldg(g.pairs + t);
    c.kind = 1, c.len = 2, c.idx[0] = p.x, c.idx[1] = p.y;
    c.masked = g.pair_masked ? g.pair_masked[t] : 0;
    return;
  }
  long q = t - g.npairs;
  if (q < g.nseg) {
    const int a = __ldg(g.seg_ptr + q), b = __ldg(g.seg_ptr + q + 1);
    if (b - a > kGsCache) {
      c.kind = 4;
      return;
    }
    c.kind = 2, c.len = b - a;
    for (int k = 0; k < b - a; k++) c.idx[k] = __ldg(g.seg_idx + a + k);
    c.masked = g.seg_masked ? g.seg_masked[q] : 0;
    return;
  }
  q -= g.nseg;
  c.kind = 3, c.len = 1, c.idx[0] = __ldg(g.extra_mask + q);
}

// gs_add_item (with mask, no scale) on a cached item: the same sums in the
// same order.
__device__ __forceinline__ void gs_cached_add(double *__restrict__ u, const GsSlot &c) {
  if (c.kind == 1) {
    double s = u[c.idx[0]] + u[c.idx[1]];
    if (c.masked) s = 0.0;
    u[c.idx[0]] = s;
    u[c.idx[1]] = s;
  } else if (c.kind == 2) {
    double v[kGsCache];
#pragma unroll
    for (int k = 0; k < kGsCache; k++) v[k] = k < c.len ? u[c.idx[k]] : 0.0;
    double s = v[0];
#pragma unroll
    for (int k = 1; k < kGsCache; k++)
      if (k < c.len) s = s + v[k];
    if (c.masked) s = 0.0;
#pragma unroll
    for (int k = 0; k < kGsCache; k++)
      if (k < c.len) u[c.idx[k]] = s;
  } else if (c.kind == 3) {
    u[c.idx[0]] = 0.0;
  }
}

// REGS: every thread's points fit in one chunk and x, r, z, p stay in registers;
// otherwise they are read and written chunk by chunk.
template <bool REGS>
__global__ void __launch_bounds__(kCoarseThreads) coarse_cg_grid_kernel(const CoarseCg a) {
  if (a.skip && *a.skip) return;
  __shared__ double sD[4], sDt[4];
  __shared__ GsSlot gslot[kCoarseThreads];
  const long nc = a.nelv * 8;
  const long stride = (long)gridDim.x * kCoarseThreads;
  const long t0 = (long)blockIdx.x * kCoarseThreads + threadIdx.x;
  const int lane = threadIdx.x & 31;
  if (threadIdx.x < 4) {
    sD[threadIdx.x] = a.D[threadIdx.x];
    sDt[threadIdx.x] = a.Dt[threadIdx.x];
  }
  const long nitems = gs_items(a.gs, true);
  gs_cache_item(gslot[threadIdx.x], a.gs, t0);
  __syncthreads();
  int buf = 0;
  auto allsum2 = [&](double v0, double v1, double &s0, double &s1) {
    const bool ok = grid_allsum2(v0, v1, a.part + (size_t)buf * 2 * gridDim.x, a.bar, a.err,
                                 s0, s1);
    buf ^= 1;
    return ok;
  };
  // gs + mask: the first item from the cache, further ones (more items
  // than threads) as usual
  auto gs_phase = [&](double *u) {
    const GsSlot &c = gslot[threadIdx.x];
    if (c.kind == 4)
      gs_add_item<double>(u, a.gs, (int)t0, true, nullptr);
    else
      gs_cached_add(u, c);
    for (long t = t0 + stride; t < nitems; t += stride)
      gs_add_item<double>(u, a.gs, (int)t, true, nullptr);
  };
  gs_phase(a.f);
  if (!grid_barrier(a.bar, a.err)) return;

  // Point loops run in chunks of points per thread with every load of a chunk
  // issued before its first use; sums follow the points in order.
  double x[kU], r[kU], z[kU], p[kU];
  double s_rr = 0.0, s_rz = 0.0;
  for (long q0 = t0; q0 < nc; q0 += kU * stride) {
    double m[kU], dv[kU];
#pragma unroll
    for (int u = 0; u < kU; u++) {
      const long q = q0 + u * stride;
      const bool ok = q < nc;
      r[u] = ok ? a.f[q] : 0.0;
      m[u] = ok ? __ldg(a.mult + q) : 0.0;
      dv[u] = ok ? __ldg(a.dinv + q) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < kU; u++) {
      const long q = q0 + u * stride;
      x[u] = p[u] = z[u] = 0.0;
      if (q < nc) {
        z[u] = __dmul_rn(r[u], dv[u]);  // rounded here whatever uses it
        if (!REGS) {
          a.x[q] = 0.0;
          a.p[q] = 0.0;
          a.r[q] = r[u];
          a.z[q] = z[u];
        }
        s_rr += r[u] * m[u] * r[u];
        s_rz += r[u] * m[u] * z[u];
      }
    }
    if (REGS) break;
  }
  double rtr, rtz;
  if (!allsum2(s_rr, s_rz, rtr, rtz)) return;
  double rn = sqrt(rtr) * a.norm_fac;
  bool done = fabs(rn) < 2.220446049250313e-16;
  int iter = 0;
  double rtz_old = 1.0;

  while (!done) {
    const double beta = iter == 0 ? 0.0 : rtz / rtz_old;
    // p = z + beta p; w = A p (local); (p, w_local)
    double s_pw = 0.0;
    auto ax_chunk = [&](long qb0, double *pu, const double *zu) {
      double H[kUA], G11[kUA], G22[kUA], G33[kUA], G12[kUA], G13[kUA], G23[kUA];
#pragma unroll
      for (int u = 0; u < kUA; u++) {
        const long q = qb0 + u * stride + lane;
        const bool act = q < nc;
        H[u] = act ? __ldg(a.h1 + q) : 0.0;
        G11[u] = act ? __ldg(a.g[0] + q) : 0.0;
        G22[u] = act ? __ldg(a.g[1] + q) : 0.0;
        G33[u] = act ? __ldg(a.g[2] + q) : 0.0;
        G12[u] = act ? __ldg(a.g[3] + q) : 0.0;
        G13[u] = act ? __ldg(a.g[4] + q) : 0.0;
        G23[u] = act ? __ldg(a.g[5] + q) : 0.0;
      }
#pragma unroll
      for (int u = 0; u < kUA; u++) {
        const long qb = qb0 + u * stride;
        if (qb >= nc) break;  // warp-uniform: qb is the warp's first point
        const long q = qb + lane;
        const bool act = q < nc;
        pu[u] = act ? zu[u] + beta * pu[u] : 0.0;
        const double wq =
            ax_lx2(pu[u], lane, sD, sDt, H[u], G11[u], G22[u], G33[u], G12[u], G13[u], G23[u]);
        if (act) {
          a.w[q] = wq;
          s_pw += pu[u] * wq;
        }
      }
    };
    if (REGS) {
#pragma unroll
      for (int h = 0; h < kU; h += kUA)
        if (t0 - lane + h * stride < nc) ax_chunk(t0 - lane + h * stride, p + h, z + h);
    } else {
      for (long qb0 = t0 - lane; qb0 < nc; qb0 += kUA * stride) {
        double pq[kUA], zq[kUA];
#pragma unroll
        for (int u = 0; u < kUA; u++) {
          const long q = qb0 + u * stride + lane;
          zq[u] = q < nc ? a.z[q] : 0.0;
          pq[u] = q < nc ? a.p[q] : 0.0;
        }
        ax_chunk(qb0, pq, zq);
#pragma unroll
        for (int u = 0; u < kUA; u++) {
          const long q = qb0 + u * stride + lane;
          if (q < nc) a.p[q] = pq[u];
        }
      }
    }
    double pap, unused;
    if (!allsum2(s_pw, 0.0, pap, unused)) return;
    const double alpha = rtz / pap;
    gs_phase(a.w);
    if (!grid_barrier(a.bar, a.err)) return;
    // x += alpha p; r -= alpha w; z = d r; (r, mult r), (r, mult z)
    s_rr = 0.0;
    s_rz = 0.0;
    const double malpha = -alpha;
    for (long q0 = t0; q0 < nc; q0 += kU * stride) {
      double wq[kU], m[kU], dv[kU];
#pragma unroll
      for (int u = 0; u < kU; u++) {
        const long q = q0 + u * stride;
        const bool ok = q < nc;
        wq[u] = ok ? a.w[q] : 0.0;
        m[u] = ok ? __ldg(a.mult + q) : 0.0;
        dv[u] = ok ? __ldg(a.dinv + q) : 0.0;
        if (!REGS) {
          x[u] = ok ? a.x[q] : 0.0;
          p[u] = ok ? a.p[q] : 0.0;
          r[u] = ok ? a.r[q] : 0.0;
        }
      }
#pragma unroll
      for (int u = 0; u < kU; u++) {
        const long q = q0 + u * stride;
        if (q < nc) {
          x[u] = x[u] + alpha * p[u];
          r[u] = r[u] + malpha * wq[u];
          z[u] = __dmul_rn(r[u], dv[u]);
          if (!REGS) {
            a.x[q] = x[u];
            a.r[q] = r[u];
            a.z[q] = z[u];
          }
          s_rr += r[u] * m[u] * r[u];
          s_rz += r[u] * m[u] * z[u];
        }
      }
      if (REGS) break;
    }
    double rtz_new;
    if (!allsum2(s_rr, s_rz, rtr, rtz_new)) return;
    rtz_old = rtz;
    rtz = rtz_new;
    rn = sqrt(rtr) * a.norm_fac;
    iter += 1;
    done = !(rn == rn) || isinf(rn) || rn < a.tol || iter >= a.niter;
  }
  if (REGS) {
#pragma unroll
    for (int u = 0; u < kU; u++) {
      const long q = t0 + u * stride;
      if (q < nc) a.x[q] = x[u];
    }
  }
}

template <bool REGS>
static cudaError_t launch_coarse_grid(const CoarseCg &a, int grid, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(kCoarseThreads);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;  // its blocks wait on one another
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, coarse_cg_grid_kernel<REGS>, a);
}

template <typename T>
cudaError_t hsmg_coarse_restrict(const CoarseArgs<T> &a, int lm, const int *skip,
                                 cudaStream_t s, bool chain) {
  const long nc = a.nelv * 8, points = chain ? nc : kNotChained;
  const unsigned grid = (unsigned)((nc + 255) / 256);
  switch (lm) {
    case 3:
      launch_chained(points, coarse_restrict_kernel<T, 3>, grid, 256, 0, s, a.w_mid, a.mult_m, a.J,
                     a.f, nc, skip);
      break;
    case 4:
      launch_chained(points, coarse_restrict_kernel<T, 4>, grid, 256, 0, s, a.w_mid, a.mult_m, a.J,
                     a.f, nc, skip);
      break;
    default: return cudaErrorNotSupported;
  }
  return cudaGetLastError();
}
template cudaError_t hsmg_coarse_restrict<double>(const CoarseArgs<double> &, int, const int *,
                                                  cudaStream_t, bool);
template cudaError_t hsmg_coarse_restrict<float>(const CoarseArgs<float> &, int, const int *,
                                                 cudaStream_t, bool);

static cudaError_t resident_limit(int &limit) {
  static int known[64];
  return cluster_limit(coarse_cg_resident_kernel, kCoarseStageBytes, known, limit);
}

cudaError_t hsmg_coarse_nodes(int &most) {
  int limit = 0;
  const cudaError_t e = resident_limit(limit);
  most = limit * kCoarseThreads;
  return e;
}

cudaError_t hsmg_coarse_cg(const CoarseCg &a, const int *skip, cudaStream_t s) {
  const NodeOp &A = a.A;
  if (A.nn == 0) return cudaSuccess;  // every vertex masked: no correction
  CoarseCg b = a;
  b.skip = skip;
  int limit = 0, nblk = 1;
  cudaError_t e;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at[3];
  if (A.val) {  // assembled: z, p and, where it fits, the matrix resident
    if ((e = resident_limit(limit)) != cudaSuccess) return e;
    while (nblk < limit && nblk * kCoarseRowsPerBlock < A.nn) nblk *= 2;
    const int slices = (A.ns + nblk - 1) / nblk;
    const size_t slice = (size_t)A.maxw * 32 * (sizeof(double) + sizeof(int)),
                 vectors = 2 * (size_t)A.nn * sizeof(double);
    b.stage_slices = vectors + slices * slice <= kCoarseStageBytes ? slices : 0;
    cluster_config(cfg, at, nblk, vectors + b.stage_slices * slice, s, 8L * a.nelv,
                   a.priority);
    return cudaLaunchKernelEx(&cfg, coarse_cg_resident_kernel, b);
  }
  // element-local: a block for every 512 points of the middle level, at most one
  // a multiprocessor (co-resident, few arrivals)
  const long work = a.nelv * a.lm * a.lm * a.lm;
  long g = (work + kCoarseThreads - 1) / kCoarseThreads;
  if (g > device_sms()) g = device_sms();
  if (g > kCoarseMaxBlocks) g = kCoarseMaxBlocks;
  return a.nelv * 8 <= kU * g * kCoarseThreads ? launch_coarse_grid<true>(b, (int)g, s)
                                               : launch_coarse_grid<false>(b, (int)g, s);
}

}  // namespace nb

// ---------------------------------------------------------------------------
// Self-test of the bounded waits: each probe waits on something that never
// happens -- a grid barrier that one of two blocks skips, an mbarrier that
// nothing arrives on -- with a short poll limit, and must come back with
// its timeout flag set instead of hanging.
// ---------------------------------------------------------------------------
namespace nb {

__global__ void barrier_timeout_probe(unsigned *bar, int *err) {
  if (blockIdx.x == 1) return;  // never arrives
  grid_barrier(bar, err, 1u << 14);
}

__global__ void mbarrier_timeout_probe(int *out) {
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    fence_barrier_init();
  }
  __syncthreads();
  const bool ok = mbar_wait(&bar, 0, 1 << 12);  // nothing arrives
  if (threadIdx.x == 0) *out = ok ? 0 : 1;
  __syncthreads();
  if (threadIdx.x == 0) {  // complete the phase so the barrier is left at rest
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(&bar)) : "memory");
  }
}

}  // namespace nb

extern "C" nb_status nb_selftest_bounded_waits(int *barrier_timed_out, int *mbarrier_timed_out) {
  using namespace nb;
  if (!barrier_timed_out || !mbarrier_timed_out) {
    set_error("null argument");
    return NB_ERR_ARG;
  }
  int *buf = nullptr;  // bar, err, mbarrier result
  cudaError_t e = cudaMalloc(&buf, 4 * sizeof(int));
  if (e == cudaSuccess) e = cudaMemset(buf, 0, 4 * sizeof(int));
  if (e == cudaSuccess) {
    barrier_timeout_probe<<<2, 32>>>(reinterpret_cast<unsigned *>(buf), buf + 1);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) {
    mbarrier_timeout_probe<<<1, 32>>>(buf + 2);
    e = cudaGetLastError();
  }
  int h[4] = {0, 0, 0, 0};
  if (e == cudaSuccess) e = cudaMemcpy(h, buf, sizeof(h), cudaMemcpyDeviceToHost);
  cudaFree(buf);
  if (e != cudaSuccess) {
    set_error(std::string("selftest: ") + cudaGetErrorString(e));
    return NB_ERR_CUDA;
  }
  *barrier_timed_out = h[1];
  *mbarrier_timed_out = h[2];
  return NB_OK;
}
