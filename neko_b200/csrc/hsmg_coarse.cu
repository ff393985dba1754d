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
// owns it, the matrix in the shared memory of its block when it fits.  Up to
// 8192 vertices each block also holds all of z and p in shared memory: a
// thread sends its z to every block before the barrier of the sums, and each
// block forms p for itself, which leaves two cluster barriers an iteration
// and gathers that never leave the block.  Beyond, p is exchanged through
// global memory at the price of a third barrier.
//
// A solve on 343 vertices (8^3 elements) took 124 us as a cooperative grid
// with barriers in global memory and element-local vectors (33 barriers of
// about 3.7 us with their sums), 67 us with p in global memory.
// A cluster leaves the other multiprocessors to the fine-level smoother,
// which runs beside it; the grid form held one block on every one.
//
// The arithmetic is that of cg_init / cg_precond_dot / cg_update_p /
// ax_helm / gs / cg_update_xr with sums over distinct points: a mult-weighted
// sum over the copies of a point is one term here, and (p, w) of the
// assembled operator is the reference's (p, mult gs(w)).
#include <cmath>
#include <string>

#include "nb_cluster.cuh"
#include "nb_nodes.h"
#include "nb_precond.h"
#include "nb_reduce.cuh"
#include "nb_tma.cuh"

namespace nb {

// rows a block aims at when the cluster grows: below, the block's own work is
// shorter than a larger cluster's barrier
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

// one slice of the matrix to shared memory
__device__ __forceinline__ void stage_slice(const NodeOp &A, int s, double *val, int *col,
                                            int lane) {
  const int o = __ldg(A.soff + s), w = __ldg(A.soff + s + 1) - o;
  const double *gv = A.val + 32 * (size_t)o + lane;
  const int *gc = A.col + 32 * (size_t)o + lane;
#pragma unroll 9
  for (int k = 0; k < w; k++) {
    val[32 * k + lane] = __ldg(gv + 32 * k);
    col[32 * k + lane] = __ldg(gc + 32 * k);
  }
}

// The solve with at most one row a thread (8192 vertices): all of z and p in
// every block's shared memory.
__global__ void __launch_bounds__(kCoarseThreads) coarse_cg_resident_kernel(const CoarseCg a) {
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

// The solve on more vertices: p exchanged through global memory.  Warp t of
// the cluster takes matrix slices t, t + warps, ...; with RPT > 0 a thread
// owns at most RPT rows and keeps their vectors in registers, with RPT = 0
// (more rows than that) they are kept in global memory.
template <int RPT>
__global__ void __launch_bounds__(kCoarseThreads)
    coarse_cg_kernel(const CoarseCg a) {
  if (a.skip && *a.skip) return;
  constexpr int NR = RPT > 0 ? RPT : 1;
  extern __shared__ __align__(16) unsigned char coarse_smem[];
  __shared__ ClusterSums sums;
  const NodeOp &A = a.A;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const unsigned rank = cluster_rank(), nblk = gridDim.x;
  const int warps = kCoarseWarps * (int)nblk, first = wid * (int)nblk + (int)rank;
  double x[NR], r[NR], z[NR], p[NR], d[NR];

  // calls body(s, row, x, r, z, p, d) for each row of this thread
  auto rows = [&](auto &&body) {
    if constexpr (RPT > 0) {
#pragma unroll
      for (int j = 0; j < RPT; j++) {
        const int s = first + j * warps, row = 32 * s + lane;
        if (row < A.nn) body(j, s, row, x[j], r[j], z[j], p[j], d[j]);
      }
    } else {
      int j = 0;
      for (int s = first; s < A.ns; s += warps, j++) {
        const int row = 32 * s + lane;
        if (row >= A.nn) continue;
        double xv = a.x[row], rv = a.r[row], dv = A.dinv[row], pv = __ldcg(a.p + row);
        double zv = dv * rv;
        body(j, s, row, xv, rv, zv, pv, dv);
        a.x[row] = xv;
        a.r[row] = rv;
      }
    }
  };

  // this block's slices of the matrix in shared memory, at a common pitch
  double *sval = reinterpret_cast<double *>(coarse_smem);
  int *scol = reinterpret_cast<int *>(sval + (size_t)a.stage_slices * A.maxw * 32);
  if (a.stage_slices > 0) {
    int j = 0;
    for (int s = first; s < A.ns; s += warps, j++) {
      const size_t to = (size_t)(j * kCoarseWarps + wid) * A.maxw * 32;
      stage_slice(A, s, sval + to, scol + to, lane);
    }
    __syncwarp();
  }
  // (A p)(row) of slice s, the j-th of this warp
  auto matvec = [&](int j, int s) {
    const int o = __ldg(A.soff + s), w = __ldg(A.soff + s + 1) - o;
    const size_t st = (size_t)(j * kCoarseWarps + wid) * A.maxw * 32 + lane;
    const double *val = a.stage_slices > 0 ? sval + st : A.val + 32 * (size_t)o + lane;
    const int *col = a.stage_slices > 0 ? scol + st : A.col + 32 * (size_t)o + lane;
    return row_dot(val, col, w, [&](int c) { return __ldcg(a.p + c); });
  };

  // x = 0, r = f, z = d r, p = 0; (r, r), (r, z)
  double s_rr = 0.0, s_rz = 0.0;
  if constexpr (RPT == 0) {
    for (int s = first; s < A.ns; s += warps) {
      const int row = 32 * s + lane;
      if (row < A.nn) {
        a.x[row] = 0.0;
        a.r[row] = 0.0;
        a.p[row] = 0.0;
      }
    }
  }
  rows([&](int, int, int row, double &xv, double &rv, double &zv, double &pv, double &dv) {
    xv = 0.0;
    rv = node_rhs(A, a.f, row);
    pv = 0.0;
    if (RPT > 0) dv = __ldg(A.dinv + row);
    zv = dv * rv;
    s_rr += rv * rv;
    s_rz += rv * zv;
  });
  cluster_barrier();  // every block runs before its shared memory is written to
  double rtr, rtz;
  cluster_allsum2(s_rr, s_rz, sums, 0, rank, nblk, rtr, rtz);
  double rn = sqrt(rtr) * a.norm_fac;
  bool done = fabs(rn) < 2.220446049250313e-16;
  int iter = 0;
  double rtz_old = 1.0;
  while (!done) {
    const double beta = iter == 0 ? 0.0 : rtz / rtz_old;
    rows([&](int, int, int row, double &, double &, double &zv, double &pv, double &) {
      pv = zv + beta * pv;
      a.p[row] = pv;
    });
    cluster_barrier();
    double s_pw = 0.0, w[NR];
    rows([&](int j, int s, int row, double &, double &, double &, double &pv, double &) {
      const double wv = matvec(j, s);
      if constexpr (RPT > 0)
        w[j] = wv;
      else
        a.w[row] = wv;
      s_pw += pv * wv;
    });
    double pap, unused;
    cluster_allsum2(s_pw, 0.0, sums, 1, rank, nblk, pap, unused);
    const double alpha = rtz / pap, malpha = -alpha;
    s_rr = 0.0;
    s_rz = 0.0;
    rows([&](int j, int, int row, double &xv, double &rv, double &zv, double &pv, double &dv) {
      double wv;
      if constexpr (RPT > 0)
        wv = w[j];
      else
        wv = a.w[row];
      xv = xv + alpha * pv;
      rv = rv + malpha * wv;
      zv = dv * rv;
      s_rr += rv * rv;
      s_rz += rv * zv;
    });
    double rtz_new;
    cluster_allsum2(s_rr, s_rz, sums, 0, rank, nblk, rtr, rtz_new);
    rtz_old = rtz;
    rtz = rtz_new;
    rn = sqrt(rtr) * a.norm_fac;
    iter += 1;
    done = !(rn == rn) || isinf(rn) || rn < a.tol || iter >= a.niter;
  }
  if constexpr (RPT > 0)
    rows([&](int, int, int row, double &xv, double &, double &, double &, double &) {
      a.x[row] = xv;
    });
}

template <typename T>
cudaError_t hsmg_coarse_restrict(const CoarseArgs<T> &a, int lm, const int *skip,
                                 cudaStream_t s) {
  const long nc = a.nelv * 8;
  const unsigned grid = (unsigned)((nc + 255) / 256);
  switch (lm) {
    case 3:
      coarse_restrict_kernel<T, 3><<<grid, 256, 0, s>>>(a.w_mid, a.mult_m, a.J, a.f, nc, skip);
      break;
    case 4:
      coarse_restrict_kernel<T, 4><<<grid, 256, 0, s>>>(a.w_mid, a.mult_m, a.J, a.f, nc, skip);
      break;
    default: return cudaErrorNotSupported;
  }
  return cudaGetLastError();
}
template cudaError_t hsmg_coarse_restrict<double>(const CoarseArgs<double> &, int, const int *,
                                                  cudaStream_t);
template cudaError_t hsmg_coarse_restrict<float>(const CoarseArgs<float> &, int, const int *,
                                                 cudaStream_t);

cudaError_t hsmg_coarse_cg(const CoarseCg &a, const int *skip, cudaStream_t s) {
  if (a.A.nn == 0) return cudaSuccess;  // every vertex masked: no correction
  // resident form (one row a thread), two, four rows a thread, any number
  constexpr int kForms = 4;
  using CoarseKernel = void (*)(CoarseCg);
  static const CoarseKernel kernels[kForms] = {coarse_cg_resident_kernel, coarse_cg_kernel<2>,
                                               coarse_cg_kernel<4>, coarse_cg_kernel<0>};
  static const int rows[kForms] = {1, 2, 4, 0};
  static int known[kForms][64];
  const NodeOp &A = a.A;
  const size_t slice = (size_t)A.maxw * 32 * (sizeof(double) + sizeof(int));
  for (int v = 0; v < kForms; v++) {
    int limit = 0, nblk = 1;
    cudaError_t e = cluster_limit(kernels[v], kCoarseStageBytes, known[v], limit);
    if (e != cudaSuccess) return e;
    while (nblk < limit && nblk * kCoarseRowsPerBlock < A.nn) nblk *= 2;
    const int per_block = (A.ns + nblk - 1) / nblk;
    const int per_warp = (per_block + kCoarseWarps - 1) / kCoarseWarps;
    if (rows[v] > 0 && per_warp > rows[v]) continue;
    const size_t vectors = v == 0 ? 2 * (size_t)A.nn * sizeof(double) : 0;
    CoarseCg b = a;
    b.skip = skip;
    // slices at a common pitch, warp by warp
    const int staged = per_warp > 1 ? per_warp * kCoarseWarps : per_block;
    b.stage_slices = vectors + staged * slice <= kCoarseStageBytes ? staged : 0;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at;
    cluster_config(cfg, at, nblk, vectors + b.stage_slices * slice, s);
    return cudaLaunchKernelEx(&cfg, kernels[v], b);
  }
  return cudaErrorNotSupported;
}

}  // namespace nb

// ---------------------------------------------------------------------------
// Self-test of the bounded waits: each probe waits on something that never
// happens -- a grid barrier that one of two blocks skips, an mbarrier that
// nothing arrives on -- with a short poll limit, and must come back with
// its timeout flag set instead of hanging.
// ---------------------------------------------------------------------------
namespace nb {

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
