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
// with three barriers (|).  The whole solve is one thread-block cluster (up
// to 16 blocks on one GPC): its barriers are hardware barriers, and its
// sums travel through distributed shared memory.  The vectors of a row stay
// in the registers of the thread that owns it, the matrix in the shared
// memory of its block when it fits.  A solve on 4096 vertices took 124 us as
// a cooperative grid with barriers in global memory and element-local
// vectors (33 barriers of about 3.7 us with their sums).  A cluster leaves the
// other multiprocessors to the fine-level smoother, which runs beside it;
// the grid form held one block on every one.
//
// The arithmetic is that of cg_init / cg_precond_dot / cg_update_p /
// ax_helm / gs / cg_update_xr with sums over distinct points: a mult-weighted
// sum over the copies of a point is one term here, and (p, w) of the
// assembled operator is the reference's (p, mult gs(w)).
#include <cmath>
#include <string>

#include "nb_nodes.h"
#include "nb_precond.h"
#include "nb_reduce.cuh"
#include "nb_tma.cuh"

namespace nb {

constexpr int kCoarseThreads = 512;
constexpr int kCoarseWarps = kCoarseThreads / 32;
constexpr int kMaxCluster = 16;
// rows a block aims at when the cluster grows: below, the block's own work is
// shorter than a larger cluster's barrier
constexpr int kCoarseRowsPerBlock = 256;
// shared memory a block may spend on its part of the matrix
constexpr size_t kCoarseStageBytes = 160 * 1024;

__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// All threads of the cluster; orders their global and shared writes.
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::
                   : "memory");
}
// *p = v in the shared memory of block `rank` of the cluster (p: this
// block's address of the variable).
__device__ __forceinline__ void cluster_store(double *p, unsigned rank, double v) {
  unsigned a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_addr(p)), "r"(rank));
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

// Two sums over the cluster, identical in every thread: block sums, sent to
// every block's slot of this block, a barrier, then each warp adds the slots
// in one fixed tree.  Consecutive calls alternate `slots`.
struct ClusterSums {
  double slot[2][kMaxCluster][2];
  double warp[kCoarseWarps][2];
};
__device__ __forceinline__ void cluster_allsum2(double v0, double v1, ClusterSums &sm, int buf,
                                                unsigned rank, unsigned nblk, double &t0,
                                                double &t1) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  v0 = warp_sum(v0);
  v1 = warp_sum(v1);
  if (lane == 0) {
    sm.warp[wid][0] = v0;
    sm.warp[wid][1] = v1;
  }
  __syncthreads();
  if (wid == 0) {
    v0 = lane < kCoarseWarps ? sm.warp[lane][0] : 0.0;
    v1 = lane < kCoarseWarps ? sm.warp[lane][1] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      v0 += __shfl_xor_sync(0xffffffffu, v0, o);
      v1 += __shfl_xor_sync(0xffffffffu, v1, o);
    }
    if (lane < (int)nblk) {
      cluster_store(&sm.slot[buf][rank][0], lane, v0);
      cluster_store(&sm.slot[buf][rank][1], lane, v1);
    }
  }
  cluster_barrier();
  t0 = lane < (int)nblk ? sm.slot[buf][lane][0] : 0.0;
  t1 = lane < (int)nblk ? sm.slot[buf][lane][1] : 0.0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    t0 += __shfl_xor_sync(0xffffffffu, t0, o);
    t1 += __shfl_xor_sync(0xffffffffu, t1, o);
  }
}

// f(o,p,r) = sum_k J(k,r) sum_j J(j,p) sum_i J(i,o) (w mult)(i,j,k) per
// element, in T and in the order of tensor3_kernel (x, then y, then z); one
// thread a vertex of an element.
template <typename T, int LM>
__global__ void __launch_bounds__(256)
    coarse_restrict_kernel(const T *__restrict__ w_mid, const T *__restrict__ mult_m,
                           const T *__restrict__ J, double *__restrict__ f, long nc,
                           const int *__restrict__ skip) {
  if (skip && *skip) return;
  constexpr int M3 = LM * LM * LM;
  __shared__ T sJ[LM * 2];  // J(m, c) at m + LM c
  if (threadIdx.x < LM * 2) sJ[threadIdx.x] = J[threadIdx.x];
  __syncthreads();
  const long q = blockIdx.x * 256L + threadIdx.x;
  if (q >= nc) return;
  const long e = q >> 3;
  const int o = q & 1, pp = (q >> 1) & 1, rr = (q >> 2) & 1;
  const T *in = w_mid + e * M3, *sc = mult_m + e * M3;
  T acc_z = 0;
#pragma unroll
  for (int k = 0; k < LM; k++) {
    T acc_y = 0;
#pragma unroll
    for (int j = 0; j < LM; j++) {
      T acc_x = 0;
#pragma unroll
      for (int i = 0; i < LM; i++) {
        const int m = i + LM * (j + LM * k);
        acc_x += sJ[i + LM * o] * (T)(__ldg(in + m) * __ldg(sc + m));
      }
      acc_y += sJ[j + LM * pp] * acc_x;
    }
    acc_z += sJ[k + LM * rr] * acc_y;
  }
  f[q] = (double)acc_z;
}

// niter Jacobi-CG iterations (or to the absolute tolerance) of A x = f from
// zero, f the sum of the element-local `a.f` over a node's copies.  Warp t
// of the cluster takes matrix slices t, t + warps, ...; with RPT > 0 a thread
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
      const int o = __ldg(A.soff + s), w = __ldg(A.soff + s + 1) - o;
      const size_t to = (size_t)(j * kCoarseWarps + wid) * A.maxw * 32 + lane;
      for (int k = 0; k < w; k++) {
        sval[to + 32 * k] = __ldg(A.val + 32 * ((size_t)o + k) + lane);
        scol[to + 32 * k] = __ldg(A.col + 32 * ((size_t)o + k) + lane);
      }
    }
    __syncwarp();
  }
  // (A p)(row) of slice s, the j-th of this warp: nine entries at a time (a
  // third of a box row), their vector values in flight together
  auto matvec = [&](int j, int s) {
    const int o = __ldg(A.soff + s), w = __ldg(A.soff + s + 1) - o;
    const size_t st = (size_t)(j * kCoarseWarps + wid) * A.maxw * 32 + lane;
    const double *val = a.stage_slices > 0 ? sval + st : A.val + 32 * (size_t)o + lane;
    const int *col = a.stage_slices > 0 ? scol + st : A.col + 32 * (size_t)o + lane;
    double acc = 0.0;
    int k = 0;
    for (; k + 9 <= w; k += 9) {
      double v[9];
#pragma unroll
      for (int u = 0; u < 9; u++) v[u] = __ldcg(a.p + col[32 * (k + u)]);
#pragma unroll
      for (int u = 0; u < 9; u++) acc += val[32 * (k + u)] * v[u];
    }
    for (; k < w; k++) acc += val[32 * k] * __ldcg(a.p + col[32 * k]);
    return acc;
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
    double f = 0.0;
    for (int k = __ldg(A.eptr + row); k < __ldg(A.eptr + row + 1); k++)
      f += a.f[__ldg(A.ent + k)];
    xv = 0.0;
    rv = f;
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

// Blocks of the largest cluster the device takes for this kernel: 16 (one
// GPC, an opt-in size) where it is accepted, else the portable 8.
template <int RPT>
static cudaError_t cluster_limit(int &limit) {
  static int known[64] = {0};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  int &k = known[dev & 63];
  if (k == 0) {
    auto kern = coarse_cg_kernel<RPT>;
    if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)kCoarseStageBytes)) != cudaSuccess)
      return e;
    k = 8;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
        cudaSuccess) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(kMaxCluster);
      cfg.blockDim = dim3(kCoarseThreads);
      cfg.dynamicSmemBytes = kCoarseStageBytes;
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = kMaxCluster;
      at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
      cfg.attrs = at;
      cfg.numAttrs = 1;
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess && n >= 1) k = kMaxCluster;
    }
    cudaGetLastError();  // a refused cluster size is not an error of the caller
  }
  limit = k;
  return cudaSuccess;
}

template <int RPT>
static cudaError_t launch_cg(CoarseCg a, int nblk, cudaStream_t s) {
  const int warps = kCoarseWarps * nblk, per_warp = (a.A.ns + warps - 1) / warps;
  const size_t bytes = (size_t)per_warp * kCoarseWarps * a.A.maxw * 32 * (sizeof(double) + sizeof(int));
  a.stage_slices = bytes <= kCoarseStageBytes ? per_warp * kCoarseWarps : 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)nblk);
  cfg.blockDim = dim3(kCoarseThreads);
  cfg.dynamicSmemBytes = a.stage_slices ? bytes : 0;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)nblk;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, coarse_cg_kernel<RPT>, a);
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
  CoarseCg b = a;
  b.skip = skip;
  int limit = 0;
  cudaError_t e = cluster_limit<1>(limit);
  if (e != cudaSuccess) return e;
  int nblk = 1;
  while (nblk < limit && nblk * kCoarseRowsPerBlock < a.A.nn) nblk *= 2;
  const int per_thread = (a.A.ns + kCoarseWarps * nblk - 1) / (kCoarseWarps * nblk);
  if (per_thread <= 1) return launch_cg<1>(b, nblk, s);
  if (per_thread <= 2) {
    if ((e = cluster_limit<2>(limit)) != cudaSuccess) return e;
    if (nblk <= limit) return launch_cg<2>(b, nblk, s);
  } else if (per_thread <= 4) {
    if ((e = cluster_limit<4>(limit)) != cudaSuccess) return e;
    if (nblk <= limit) return launch_cg<4>(b, nblk, s);
  }
  if ((e = cluster_limit<0>(limit)) != cudaSuccess) return e;
  return launch_cg<0>(b, nblk < limit ? nblk : limit, s);
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
