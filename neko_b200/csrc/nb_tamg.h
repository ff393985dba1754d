// nb_tamg.h -- operands of the tree-AMG cycle launch (tamg_cluster.cu).
#pragma once

#include "nb_nodes.h"

namespace nb {

// Level 0: the distinct vertices.  Level l >= 1: one entry an aggregate.
struct TamgClusterLevel {
  int n = 0;
  const int *agg = nullptr;                   // l >= 2: element -> aggregate (l = 1: itself)
  const int *sptr = nullptr, *sidx = nullptr; // l >= 1: aggregate -> vertices of its points (-1 masked)
  const int *rptr = nullptr, *ridx = nullptr; // l >= 2: aggregate -> entries of level l - 1
  const int *spread = nullptr;                // l >= 2: entry of level l - 1 -> aggregate
  double *x = nullptr, *b = nullptr, *r = nullptr, *d[2] = {nullptr, nullptr};
  double tha = 0.0, dlt = 0.0;
};
struct TamgCluster {
  NodeOp A;
  const double *mean = nullptr;       // 1 / copies of each vertex
  const TamgClusterLevel *lv = nullptr;  // device array of nlvls
  int nlvls = 0, degree = 0, cycles = 0;
  double *wn = nullptr, *yn = nullptr;   // work on the vertices
  const double *rhs = nullptr;           // element-local, assembled and masked
  double *z = nullptr;                   // element-local result
  long npts = 0;
  int nelv = 0, copies = 0;  // elements; most copies of a vertex
  int stage_slices = 0;      // set by the launch
  const int *skip = nullptr;
};
// Vertices up to which the cycle is one launch: one a thread of the largest
// cluster (8192; 4096 where the device takes clusters of the portable size
// only).  Up to there it takes 0.60 to 0.90 of the time of an application with
// the separate launches (266 against 439 us on 8^3 elements of lx 6, 609 against
// 777 on 18^3, 867 against 960 on 21^3, 8000 vertices).  Beyond, the lists and
// the matrix come from L2 in every step, to 16 multiprocessors of 148: 1.23
// against 1.22 ms on 24^3 elements, 1.71 against 1.60 on 27^3, 2.58 against 2.31
// on 32^3, 4.78 against 4.03 on 40^3.
cudaError_t tamg_cycle_nodes(int &most);
// z = `cycles` V-cycles from zero for the right-hand side rhs.
cudaError_t tamg_cycle(const TamgCluster &a, const int *skip, cudaStream_t s);

}  // namespace nb
