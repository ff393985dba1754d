// nb_cluster.cuh -- one thread-block cluster as a small machine: barrier,
// sums through distributed shared memory, sliced sparse rows and the launch.
// The coarse levels of the multigrid preconditioners run in it: their steps
// are a fraction of a microsecond, so what counts is the latency between
// them, and a hardware cluster barrier is several times shorter than one in
// global memory or a kernel boundary.
#pragma once

#include <cuda_runtime.h>

#include "nb_chain.cuh"
#include "nb_nodes.h"
#include "nb_tma.cuh"

namespace nb {

constexpr int kCoarseThreads = 512;
constexpr int kCoarseWarps = kCoarseThreads / 32;
constexpr int kMaxCluster = 16;

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

// Two sums over the cluster, identical in every thread: the warps' sums go to
// every block's slots, then each warp adds all slots in one fixed order.
// Consecutive calls alternate `buf`.  Lanes 0-15 carry the first sum, lanes
// 16-31 the second.
struct ClusterSums {
  double slot[2][kMaxCluster][kCoarseWarps][2];
};
__device__ __forceinline__ double half_warp_sum(double a) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
  return a;
}
__device__ __forceinline__ void cluster_allsum2(double v0, double v1, ClusterSums &sm, int buf,
                                                unsigned rank, unsigned nblk, double &t0,
                                                double &t1) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, h = lane >> 4, b = lane & 15;
  double a = h ? v1 : v0;
  a += __shfl_xor_sync(0xffffffffu, h ? v0 : v1, 16);
  a = half_warp_sum(a);
  if (b < (int)nblk) cluster_store(&sm.slot[buf][rank][wid][h], b, a);
  cluster_barrier();
  a = 0.0;
  for (int k = 0; k < (int)nblk; k++) a += sm.slot[buf][k][b][h];
  a = half_warp_sum(a);
  t0 = __shfl_sync(0xffffffffu, a, 0);
  t1 = __shfl_sync(0xffffffffu, a, 16);
}
static_assert(kCoarseWarps == 16, "a half-warp reads one slot of every warp");

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

// sum over the w entries of a row (stride 32) of val times load(col), nine
// entries (a third of a box row) at a time
template <typename F>
__device__ __forceinline__ double row_dot(const double *val, const int *col, int w, F &&load) {
  double acc[3] = {0.0, 0.0, 0.0};
  int k = 0;
  for (; k + 9 <= w; k += 9) {
    double v[9];
#pragma unroll
    for (int u = 0; u < 9; u++) v[u] = load(col[32 * (k + u)]);
#pragma unroll
    for (int u = 0; u < 9; u++) acc[u % 3] += val[32 * (k + u)] * v[u];
  }
  for (; k < w; k++) acc[0] += val[32 * k] * load(col[32 * k]);
  return (acc[0] + acc[1]) + acc[2];
}

// The cluster launch, at `priority` in the order of pending launches and chained
// to its predecessor in the stream when the level has few points (nb_chain.cuh).
inline void cluster_config(cudaLaunchConfig_t &cfg, cudaLaunchAttribute (&at)[3], int nblk,
                           size_t bytes, cudaStream_t s, long points, int priority = 0) {
  cfg = {};
  cfg.gridDim = dim3((unsigned)nblk);
  cfg.blockDim = dim3(kCoarseThreads);
  cfg.dynamicSmemBytes = bytes;
  cfg.stream = s;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)nblk;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributePriority;
  at[1].val.priority = priority;
  at[2].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[2].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = chained(points, s) ? 3 : 2;
}

// Blocks of the largest cluster the device takes for a kernel: 16 (one GPC,
// an opt-in size) where it is accepted with `bytes` of dynamic shared memory,
// else the portable 8.  `known` is the kernel's own record, one entry a device.
template <typename K>
cudaError_t cluster_limit(K kern, size_t bytes, int *known, int &limit) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  int &k = known[dev & 63];
  if (k == 0) {
    if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)bytes)) != cudaSuccess)
      return e;
    int best = 8;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
        cudaSuccess) {
      cudaLaunchConfig_t cfg;
      cudaLaunchAttribute at[3];
      cluster_config(cfg, at, kMaxCluster, bytes, nullptr, 0);
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess && n >= 1)
        best = kMaxCluster;
    }
    cudaGetLastError();  // a refused cluster size is not an error of the caller
    k = best;
  }
  limit = k;
  return cudaSuccess;
}

}  // namespace nb
