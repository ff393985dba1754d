// nb_nodes.h -- a vertex-level (lx = 2) problem assembled over its distinct
// points ("nodes"): the coarse level of the multigrid preconditioners.
//
// Element by element a vertex level stores every interior vertex eight
// times, and an operator application is an element kernel plus a
// gather-scatter.  Over the distinct, unmasked vertices the same operator is
// one sparse matrix (27 entries a row on a box) and the gather-scatter
// disappears, so the coarse solve needs no more than a matrix-vector product
// between two reductions.
#pragma once

#include <cuda_runtime.h>

#include <vector>

#include "nb_internal.h"

struct nb_problem;

namespace nb {

// Host-side structure, built once per level.
struct NodeHost {
  int nn = 0;                 // nodes: distinct points that are not masked
  std::vector<int> node_of;   // local point -> node, -1 on masked points
  std::vector<int> eptr, ent; // node -> its local points, ascending (CSR)
  // Matrix in slices of 32 rows (one warp's lanes), each slice padded to its
  // longest row: entry k of row 32 s + lane sits at 32 (soff[s] + k) + lane.
  std::vector<int> soff;      // slices + 1, in columns of 32 entries
  std::vector<int> col;       // padding repeats the row's own index
  std::vector<int> slot;      // 8 per entry of ent: k of each corner, -1 masked
  int maxw = 0;               // longest row
};
// maps: the level's gather-scatter maps (lx = 2, n local points); masked:
// its zero-Dirichlet points (0-based).  Beyond most_nodes only nn and node_of
// are filled.
void node_setup(const GsMaps &maps, long n, const std::vector<int> &masked, int most_nodes,
                NodeHost &H);

// The same on the device (one allocation, `base`).
struct NodeOp {
  int nn = 0, ns = 0, maxw = 0;
  const int *node_of = nullptr, *eptr = nullptr, *ent = nullptr, *soff = nullptr,
            *col = nullptr, *slot = nullptr;
  double *val = nullptr, *dinv = nullptr;  // matrix values; inverse Jacobi diagonal
  void *base = nullptr;
};
// Beyond most_nodes only A.nn is set (A.val stays null).
nb_status node_create(nb_problem *C, NodeOp &A, int most_nodes);
// Matrix values and dinv from the level's current coefficients, on stream s.
cudaError_t node_update(const nb_problem *C, const NodeOp &A, cudaStream_t s);

}  // namespace nb
