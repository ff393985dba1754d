// tamg_cluster.cu -- the tree-AMG V-cycle of phmg in one launch
// (tamg_mg_cycle_d, src/multigrid/tree_amg_multigrid.f90:423-495, with the
// Chebyshev smoother amg_device_cheby_solve).
//
// On the vertex level (lx = 2) and its aggregates every step of the cycle is
// a microsecond or less of work, and as separate launches the cycle is about
// a hundred of them (19 operator applications at the default settings, each
// with one or two gather-scatters, and the updates and transfers between):
// 350 of 636 us of device time of an application on 16^3 elements, and most
// of its 950 us with the gaps between launches.  Here it is one cluster, a
// barrier between steps.  Level 0 lives on the distinct vertices (nb_nodes.h),
// so its operator is one sparse product and the gather-scatters of the flat
// matvec (tree_amg.f90:393-509) become averages over a vertex's copies:
//
//   level 0:   w = A d
//   level l:   v_i = mean over the copies of vertex i of d[aggregate]
//              y = A v
//              w_c = sum over aggregate c's points of y_i / copies_i
//
// With at most one vertex and one element a thread (8192 of each) the index
// lists a thread walks in every step, and its block's rows of the matrix, are
// brought to shared memory once: a step is then one gather from L2 instead of
// a chain of three dependent ones (165 us a cycle on 3375 vertices without).
//
// A thread owns the same entries of a level's vectors in every step, so only
// what a product or a transfer reads from other threads needs a barrier; the
// direction d alternates between two buffers for the same reason, and the
// update x += d of a step is made in the next one (the same additions in the
// same order), when no other thread reads x any more.
#include "nb_chain.cuh"
#include "nb_cluster.cuh"
#include "nb_tamg.h"

namespace nb {

// Levels whose table fits in shared memory (deeper hierarchies read it from
// global memory), and copies of a vertex a resident list holds.
constexpr int kTamgLevels = 8, kTamgCopies = 8;
constexpr size_t kTamgStageBytes = 200 * 1024;

__global__ void __launch_bounds__(kCoarseThreads) tamg_cycle_kernel(const TamgCluster a) {
  chain();
  if (a.skip && *a.skip) return;
  extern __shared__ __align__(16) unsigned char tamg_smem[];
  __shared__ TamgClusterLevel lv_s[kTamgLevels];
  const NodeOp &A = a.A;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const TamgClusterLevel *lv = a.nlvls <= kTamgLevels ? lv_s : a.lv;
  if (a.nlvls <= kTamgLevels && tid < a.nlvls) lv_s[tid] = a.lv[tid];
  __syncthreads();
  const int nblk = (int)gridDim.x, warps = kCoarseWarps * nblk;
  const int gw = wid * nblk + (int)cluster_rank();  // warp of the cluster
  const int g = 32 * gw + lane, gs = 32 * warps;

  // resident form: the matrix slice of each warp, then lists of eight entries a
  // thread (entry u at 512 u + tid): elements of its vertex's copies, their
  // aggregates level by level, vertices of its element
  const bool res = a.stage_slices > 0;
  double *sval = reinterpret_cast<double *>(tamg_smem) + (size_t)wid * A.maxw * 32;
  int *scol = reinterpret_cast<int *>(reinterpret_cast<double *>(tamg_smem) +
                                      (size_t)a.stage_slices * A.maxw * 32) +
              (size_t)wid * A.maxw * 32;
  int *lists = reinterpret_cast<int *>(reinterpret_cast<double *>(tamg_smem) +
                                       (size_t)a.stage_slices * A.maxw * 32) +
               (size_t)a.stage_slices * A.maxw * 32 + tid;
  constexpr int LIST = kTamgCopies * kCoarseThreads;
  double mean_i = 0.0;
  int width = 0;
  if (res) {
    if (gw < A.ns) {
      width = __ldg(A.soff + gw + 1) - __ldg(A.soff + gw);
      stage_slice(A, gw, sval, scol, lane);
    }
    const int k0 = g < A.nn ? __ldg(A.eptr + g) : 0, k1 = g < A.nn ? __ldg(A.eptr + g + 1) : 0;
    const int p0 = g < lv[1].n ? __ldg(lv[1].sptr + g) : 0,
              p1 = g < lv[1].n ? __ldg(lv[1].sptr + g + 1) : 0;
    if (g < A.nn) mean_i = a.mean[g];
#pragma unroll
    for (int u = 0; u < kTamgCopies; u++) {
      const int e = k0 + u < k1 ? __ldg(A.ent + k0 + u) >> 3 : -1;
      lists[u * kCoarseThreads] = e;
      for (int l = 2; l < a.nlvls; l++)
        lists[(l - 1) * LIST + u * kCoarseThreads] = e >= 0 ? __ldg(lv[l].agg + e) : -1;
      lists[(a.nlvls - 1) * LIST + u * kCoarseThreads] =
          p0 + u < p1 ? __ldg(lv[1].sidx + p0 + u) : -1;
    }
  }
  auto list_sum = [&](const double *v, const int *q) {
    double t[kTamgCopies];
#pragma unroll
    for (int u = 0; u < kTamgCopies; u++) {
      const int k = q[u * kCoarseThreads];
      t[u] = k >= 0 ? __ldcg(v + k) : 0.0;
    }
    double acc = 0.0;
#pragma unroll
    for (int u = 0; u < kTamgCopies; u++) acc += t[u];
    return acc;
  };

  // body(i) for each entry of a level's vectors this thread owns: one thread
  // an entry on levels 0 and 1, one warp (lane 0) an aggregate above
  auto own = [&](int l, auto &&body) {
    const int n = lv[l].n;
    if (l <= 1) {
      for (int i = g; i < n; i += gs) body(i);
    } else if (lane == 0) {
      for (int i = gw; i < n; i += warps) body(i);
    }
  };
  // sum of vec over idx[p0 .. p1), by one thread
  auto gather = [&](const double *vec, const int *idx, int p0, int p1) {
    double acc = 0.0;
    for (int k = p0; k < p1; k += 8) {  // loads of eight entries in flight together
      int q[8];
      double v[8];
#pragma unroll
      for (int u = 0; u < 8; u++) q[u] = k + u < p1 ? __ldg(idx + k + u) : -1;
#pragma unroll
      for (int u = 0; u < 8; u++) v[u] = q[u] >= 0 ? __ldcg(vec + q[u]) : 0.0;
#pragma unroll
      for (int u = 0; u < 8; u++) acc += v[u];
    }
    return acc;
  };
  // the same by a warp: lanes take entries in turn, one fixed tree
  auto warp_gather = [&](const double *vec, const int *idx, int p0, int p1) {
    double acc = 0.0;
    for (int k = p0 + lane; k < p1; k += 32) {
      const int q = __ldg(idx + k);
      if (q >= 0) acc += __ldcg(vec + q);
    }
    acc = half_warp_sum(acc);
    return acc + __shfl_xor_sync(0xffffffffu, acc, 16);
  };
  // out(c) = sum over c's entries, for the owned entries of level l
  auto sums = [&](int l, const double *vec, const int *ptr, const int *idx, auto &&out) {
    const int n = lv[l].n;
    if (l == 1 && res && idx == lv[1].sidx) {
      if (g < n) out(g, list_sum(vec, lists + (a.nlvls - 1) * LIST));
    } else if (l <= 1) {
      for (int i = g; i < n; i += gs) out(i, gather(vec, idx, __ldg(ptr + i), __ldg(ptr + i + 1)));
    } else {
      for (int i = gw; i < n; i += warps) {
        const double t = warp_gather(vec, idx, __ldg(ptr + i), __ldg(ptr + i + 1));
        if (lane == 0) out(i, t);
      }
    }
  };
  // mean over the copies of vertex i of v[aggregate of the copy's element]
  auto vertex_mean = [&](int l, const double *v, int i) {
    if (res) return list_sum(v, lists + (l - 1) * LIST) * mean_i;
    const int k0 = __ldg(A.eptr + i), k1 = __ldg(A.eptr + i + 1);
    const int *agg = lv[l].agg;
    double acc = 0.0;
    for (int k = k0; k < k1; k += 8) {
      int q[8];
      double t[8];
#pragma unroll
      for (int u = 0; u < 8; u++) {
        q[u] = k + u < k1 ? __ldg(A.ent + k + u) >> 3 : -1;
        if (agg && q[u] >= 0) q[u] = __ldg(agg + q[u]);
      }
#pragma unroll
      for (int u = 0; u < 8; u++) t[u] = q[u] >= 0 ? __ldcg(v + q[u]) : 0.0;
#pragma unroll
      for (int u = 0; u < 8; u++) acc += t[u];
    }
    return acc * a.mean[i];
  };
  auto rows = [&](const double *v, auto &&out) {  // out(i, (A v)_i) on the vertices
    if (res) {
      if (g < A.nn)
        out(g, row_dot(sval + lane, scol + lane, width, [&](int c) { return __ldcg(v + c); }));
      return;
    }
    for (int s = gw; s < A.ns; s += warps) {
      const int i = 32 * s + lane;
      if (i >= A.nn) continue;
      const int o = __ldg(A.soff + s), w = __ldg(A.soff + s + 1) - o;
      const size_t at = 32 * (size_t)o + lane;
      out(i, row_dot(A.val + at, A.col + at, w, [&](int c) { return __ldcg(v + c); }));
    }
  };
  // out(i, (A_l v)_i) for the owned entries of level l
  auto matvec = [&](int l, const double *v, auto &&out) {
    cluster_barrier();  // v is complete
    if (l == 0) {
      rows(v, out);
      return;
    }
    for (int i = g; i < A.nn; i += gs) a.wn[i] = vertex_mean(l, v, i);
    cluster_barrier();
    rows(a.wn, [&](int i, double w) { a.yn[i] = w * a.mean[i]; });
    cluster_barrier();
    sums(l, a.yn, lv[l].sptr, lv[l].sidx, out);
  };
  // degree Chebyshev steps on level l for A_l x = b
  auto cheby = [&](int l, bool zero) {
    const TamgClusterLevel &L = lv[l];
    const double inv_tha = 1.0 / L.tha;
    if (zero) {
      own(l, [&](int i) {
        const double r = L.b[i];
        L.x[i] = 0.0;
        L.r[i] = r;
        L.d[0][i] = r * inv_tha;
      });
    } else {
      matvec(l, L.x, [&](int i, double w) {
        const double r = L.b[i] - w;
        L.r[i] = r;
        L.d[0][i] = r * inv_tha;
      });
    }
    const double s1 = L.tha / L.dlt;
    double rhok = 1.0 / s1;
    int cur = 0;
    for (int it = 2; it <= a.degree; it++) {
      const double rhokp1 = 1.0 / (2.0 * s1 - rhok);
      const double tmp1 = rhokp1 * rhok, tmp2 = 2.0 * rhokp1 / L.dlt;
      rhok = rhokp1;
      const double *d = L.d[cur];
      double *dn = L.d[cur ^ 1];
      matvec(l, d, [&](int i, double w) {
        const double di = d[i];
        L.x[i] = L.x[i] + di;  // the previous step's update
        const double r = L.r[i] - w;
        L.r[i] = r;
        dn[i] = tmp1 * di + tmp2 * r;
      });
      cur ^= 1;
    }
    if (l == 0 && !zero && a.degree == 1) cluster_barrier();  // x read by the only product
    const double *d = L.d[cur];
    own(l, [&](int i) { L.x[i] = L.x[i] + d[i]; });
  };

  // the right-hand side at one copy of each vertex (it is assembled)
  for (int i = g; i < A.nn; i += gs) lv[0].b[i] = a.rhs[__ldg(A.ent + __ldg(A.eptr + i))];
  const int top = a.nlvls - 1;
  for (int c = 0; c < a.cycles; c++) {
    for (int l = 0; l < top; l++) {
      cheby(l, l > 0 || c == 0);
      const TamgClusterLevel &L = lv[l], &N = lv[l + 1];
      // residual (weighted by 1 / copies on the vertices), summed over the
      // aggregates of the next level
      matvec(l, L.x, [&](int i, double w) {
        const double r = -1.0 * w + L.b[i];
        L.r[i] = l == 0 ? r * a.mean[i] : r;
      });
      cluster_barrier();
      if (l == 0)
        sums(1, L.r, N.sptr, N.sidx, [&](int i, double t) { N.b[i] = t; });
      else
        sums(l + 1, L.r, N.rptr, N.ridx, [&](int i, double t) { N.b[i] = t; });
    }
    cheby(top, true);
    for (int l = top - 1; l >= 0; l--) {
      const TamgClusterLevel &L = lv[l], &N = lv[l + 1];
      cluster_barrier();  // N.x is complete
      own(l, [&](int i) {
        const double t = l == 0 ? vertex_mean(1, N.x, i) : __ldcg(N.x + __ldg(N.spread + i));
        L.x[i] = L.x[i] + t;
      });
      cheby(l, false);
    }
  }
  // back to the element-local points
  cluster_barrier();
  for (long q = g; q < a.npts; q += gs) {
    const int i = __ldg(A.node_of + q);
    a.z[q] = i >= 0 ? __ldcg(lv[0].x + i) : 0.0;
  }
}

static cudaError_t tamg_limit(int &limit) {
  static int known[64];
  return cluster_limit(tamg_cycle_kernel, kTamgStageBytes, known, limit);
}

cudaError_t tamg_cycle_nodes(int &most) {
  int limit = 0;
  const cudaError_t e = tamg_limit(limit);
  most = limit * kCoarseThreads;
  return e;
}

cudaError_t tamg_cycle(const TamgCluster &a, const int *skip, cudaStream_t s) {
  int limit = 0, nblk = 1;
  cudaError_t e = tamg_limit(limit);
  if (e != cudaSuccess) return e;
  // a block for every 128 vertices: with 64, 128, 256 and 512 an application at lx 6
  // takes 261, 259, 265 and 283 us on 8^3 elements, 275, 273, 284 and 303 on 10^3, 475,
  // 469, 469 and 489 on 16^3
  while (nblk < limit && nblk * 128 < a.A.nn) nblk *= 2;
  TamgCluster b = a;
  b.skip = skip;
  const int threads = nblk * kCoarseThreads, slices = (a.A.ns + nblk - 1) / nblk;
  const size_t bytes = (size_t)slices * a.A.maxw * 32 * (sizeof(double) + sizeof(int)) +
                       (size_t)a.nlvls * kTamgCopies * kCoarseThreads * sizeof(int);
  const bool resident = a.A.nn <= threads && a.nelv <= threads && a.copies <= kTamgCopies &&
                        bytes <= kTamgStageBytes;
  b.stage_slices = resident ? slices : 0;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at[3];
  cluster_config(cfg, at, nblk, resident ? bytes : 0, s, a.npts);
  return cudaLaunchKernelEx(&cfg, tamg_cycle_kernel, b);
}

}  // namespace nb
