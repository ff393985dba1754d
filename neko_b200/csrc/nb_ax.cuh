// nb_ax.cuh -- shared by the translation units of the Helmholtz operator:
// ax_helm.cu (streaming forms and the entry points), ax_helm_gen.cu (general
// operator) and ax_cg_gen.cu (general fused step).  Three units, as the first use
// of a kernel loads its whole unit: in one of 15.9 MB that took 16 ms.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

#include "nb_precond.h"

namespace nb {

// Elements per block for each lx (threads = lx*lx*NE).
template <int LX>
struct AxCfg {
  static constexpr int NE = LX <= 3 ? 16 : (LX <= 5 ? 8 : (LX <= 8 ? 2 : 1));
};

// Blocks a multiprocessor that leave each thread about `regs` registers (0 in
// __launch_bounds__: the compiler's own choice).
constexpr int blocks_for(int threads, int regs) {
  const int b = 65536 / ((threads + 31) / 32 * 32 * regs);
  return b < 1 ? 1 : b;
}

// Operands; u of the plain operator, or z and p of the fused step.
template <typename TZ>
struct AxArgs {
  double *w;
  const double *u;
  double *p;
  const TZ *z;
  const double *D, *Dt, *h1, *g[6], *h2, *B;
  int nelv;
  const int *skip;
  int *err;
  // fused step
  CgState *st;
  double beta, *pap_out, *partials;
  unsigned *counter;
  int max_grid;
};

// The fused step by the general kernel, lx 2..16 (ax_cg_gen.cu).
template <typename TZ>
cudaError_t ax_cg_general(const AxArgs<TZ> &a, int lx, cudaStream_t s);

}  // namespace nb
