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
// A thread owns the same entries of a level's vectors in every step, so only
// what a product or a transfer reads from other threads needs a barrier; the
// direction d alternates between two buffers for the same reason, and the
// update x += d of a step is made in the next one (the same additions in the
// same order), when no other thread reads x any more.
#include "nb_chain.cuh"
#include "nb_cluster.cuh"
#include "nb_tamg.h"

namespace nb {

__global__ void __launch_bounds__(kCoarseThreads) tamg_cycle_kernel(const TamgCluster a) {
  chain();
  if (a.skip && *a.skip) return;
  const NodeOp &A = a.A;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int nblk = (int)gridDim.x, warps = kCoarseWarps * nblk;
  const int gw = wid * nblk + (int)cluster_rank();  // warp of the cluster
  const int g = 32 * gw + lane, gs = 32 * warps;

  // body(i) for each entry of a level's vectors this thread owns: one thread
  // an entry on levels 0 and 1, one warp (lane 0) an aggregate above
  auto own = [&](int l, auto &&body) {
    const int n = a.lv[l].n;
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
    const int n = a.lv[l].n;
    if (l <= 1) {
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
    const int k0 = __ldg(A.eptr + i), k1 = __ldg(A.eptr + i + 1);
    const int *agg = a.lv[l].agg;
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
    sums(l, a.yn, a.lv[l].sptr, a.lv[l].sidx, out);
  };
  // degree Chebyshev steps on level l for A_l x = b
  auto cheby = [&](int l, bool zero) {
    const TamgClusterLevel &L = a.lv[l];
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
  for (int i = g; i < A.nn; i += gs) a.lv[0].b[i] = a.rhs[__ldg(A.ent + __ldg(A.eptr + i))];
  const int top = a.nlvls - 1;
  for (int c = 0; c < a.cycles; c++) {
    for (int l = 0; l < top; l++) {
      cheby(l, l > 0 || c == 0);
      const TamgClusterLevel &L = a.lv[l], &N = a.lv[l + 1];
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
      const TamgClusterLevel &L = a.lv[l], &N = a.lv[l + 1];
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
    a.z[q] = i >= 0 ? __ldcg(a.lv[0].x + i) : 0.0;
  }
}

cudaError_t tamg_cycle(const TamgCluster &a, const int *skip, cudaStream_t s) {
  static int known[64];
  int limit = 0, nblk = 1;
  cudaError_t e = cluster_limit(tamg_cycle_kernel, 0, known, limit);
  if (e != cudaSuccess) return e;
  // a block for every 128 vertices, as the hsmg coarse solve
  while (nblk < limit && nblk * 128 < a.A.nn) nblk *= 2;
  TamgCluster b = a;
  b.skip = skip;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at[2];
  cluster_config(cfg, at, nblk, 0, s, a.npts);
  return cudaLaunchKernelEx(&cfg, tamg_cycle_kernel, b);
}

}  // namespace nb
