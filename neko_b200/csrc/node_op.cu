// node_op.cu -- device side of a vertex-level problem assembled over its
// distinct points (nb_nodes.h): upload of the structure and the matrix
// values.  The values are rebuilt when coefficients change, by one thread a
// row in a fixed order (the element matrices are formed on the fly), so a
// rebuild is deterministic; a thread's eight copies follow one another, 23 us on a
// small mesh.
#include <string>

#include "nb_nodes.h"
#include "nb_problem.h"

namespace nb {

// Column a of the lx = 2 element matrix of element e, the operator of
// ax_helm (+ h2 B) applied to the unit vector of corner a: col[b] = A(b, a).
// Points are (i, j, k) = bits 0, 1, 2; D is the 2 x 2 derivative matrix.
__device__ __forceinline__ void element_column(const double *D, const double *h1,
                                               const double *const g[6], const double *h2B,
                                               const double *h2, long e, int a, double col[8]) {
#pragma unroll
  for (int b = 0; b < 8; b++) col[b] = 0.0;
#pragma unroll
  for (int q = 0; q < 8; q++) {
    const int iq = q & 1, jq = (q >> 1) & 1, kq = q >> 2;
    const int ia = a & 1, ja = (a >> 1) & 1, ka = a >> 2;
    const double ur = (jq == ja && kq == ka) ? D[iq + 2 * ia] : 0.0;
    const double us = (iq == ia && kq == ka) ? D[jq + 2 * ja] : 0.0;
    const double ut = (iq == ia && jq == ja) ? D[kq + 2 * ka] : 0.0;
    const long p = 8 * e + q;
    const double H = h1[p], g11 = g[0][p], g22 = g[1][p], g33 = g[2][p], g12 = g[3][p],
                 g13 = g[4][p], g23 = g[5][p];
    const double fr = H * (g11 * ur + g12 * us + g13 * ut);
    const double fs = H * (g12 * ur + g22 * us + g23 * ut);
    const double ft = H * (g13 * ur + g23 * us + g33 * ut);
    // w(b) += D(iq, ib) fr on q's x line, and so on
#pragma unroll
    for (int v = 0; v < 2; v++) {
      col[v + 2 * jq + 4 * kq] += D[iq + 2 * v] * fr;
      col[iq + 2 * v + 4 * kq] += D[jq + 2 * v] * fs;
      col[iq + 2 * jq + 4 * v] += D[kq + 2 * v] * ft;
    }
  }
  if (h2) {
    const long p = 8 * e + a;
#pragma unroll
    for (int b = 0; b < 8; b++)
      if (b == a) col[b] += h2[p] * h2B[p];
  }
}

struct NodeCoef {
  const double *h1, *g[6], *D, *h2, *B, *jdiag;
};

// Row r of the matrix: the element rows of its copies, added in order (the
// element matrices are symmetric, so a row is the column of its corner).
__global__ void __launch_bounds__(128) node_values_kernel(NodeOp A, NodeCoef c) {
  const int r = blockIdx.x * 128 + threadIdx.x;
  if (r >= 32 * A.ns) return;
  const int s = r >> 5, lane = r & 31, w0 = A.soff[s], w = A.soff[s + 1] - w0;
  double *row = A.val + 32 * (size_t)w0 + lane;
  for (int k = 0; k < w; k++) row[32 * (size_t)k] = 0.0;
  if (r >= A.nn) return;
  double D[4];
#pragma unroll
  for (int q = 0; q < 4; q++) D[q] = c.D[q];
  for (int k = A.eptr[r]; k < A.eptr[r + 1]; k++) {
    const int p = A.ent[k];
    double v[8];
    element_column(D, c.h1, c.g, c.B, c.h2, p >> 3, p & 7, v);
#pragma unroll
    for (int b = 0; b < 8; b++) {
      const int t = A.slot[8 * (size_t)k + b];
      if (t >= 0) row[32 * (size_t)t] += v[b];
    }
  }
  A.dinv[r] = c.jdiag[A.ent[A.eptr[r]]];  // the same at every copy of a point
}

cudaError_t node_update(const nb_problem *C, const NodeOp &A, cudaStream_t s) {
  if (A.nn == 0 || !A.val) return cudaSuccess;
  const NodeCoef c{C->h1, {C->g11, C->g22, C->g33, C->g12, C->g13, C->g23}, C->D,
                   C->ifh2 ? C->h2 : nullptr, C->B, C->jdiag};
  node_values_kernel<<<(32 * A.ns + 127) / 128, 128, 0, s>>>(A, c);
  return cudaGetLastError();
}

nb_status node_create(nb_problem *C, NodeOp &A, int most_nodes) {
  std::vector<int> masked(C->nmask);
  if (C->nmask > 0)
    NB_CUDA_TRY(cudaMemcpy(masked.data(), C->msk, C->nmask * sizeof(int),
                           cudaMemcpyDeviceToHost));
  for (int &m : masked) m -= 1;
  NodeHost H;
  node_setup(C->maps, C->n, masked, most_nodes, H);
  A.nn = H.nn;
  if (A.nn > most_nodes) return NB_OK;
  A.ns = (int)H.soff.size() - 1;
  A.maxw = H.maxw;
  const std::vector<int> *src[6] = {&H.node_of, &H.eptr, &H.ent, &H.soff, &H.col, &H.slot};
  const int **dst[6] = {&A.node_of, &A.eptr, &A.ent, &A.soff, &A.col, &A.slot};
  auto slice = [](size_t bytes) { return (bytes + 255) & ~size_t(255); };
  size_t off = 0, at[6];
  for (int q = 0; q < 6; q++) {
    at[q] = off;
    off += slice(src[q]->size() * sizeof(int));
  }
  const size_t o_val = off, o_d = off + slice(H.col.size() * sizeof(double));
  const size_t bytes = o_d + slice((H.nn + 1) * sizeof(double));
  cudaError_t e = cudaMalloc(&A.base, bytes);
  if (e != cudaSuccess) {
    A.base = nullptr;
    set_error(std::string("coarse matrix: ") + cudaGetErrorString(e));
    return e == cudaErrorMemoryAllocation ? NB_ERR_OOM : NB_ERR_CUDA;
  }
  char *b = (char *)A.base;
  for (int q = 0; q < 6; q++) {
    *dst[q] = (const int *)(b + at[q]);
    if (!src[q]->empty())
      NB_CUDA_TRY(cudaMemcpy(b + at[q], src[q]->data(), src[q]->size() * sizeof(int),
                             cudaMemcpyHostToDevice));
  }
  A.val = (double *)(b + o_val);
  A.dinv = (double *)(b + o_d);
  return NB_OK;
}

}  // namespace nb
