// ax_cg_gen.cu -- the general form of the fused CG step (ax_cg_fused).
#include "nb_ax.cuh"
#include "nb_chain.cuh"
#include "nb_kernels.h"
#include "nb_precond.h"
#include "nb_reduce.cuh"

namespace nb {

// The fused step for the other orders and for operands that are not 16-byte
// aligned: NE elements a block with plain coalesced loads, the element loop of
// ax_helm_kernel.  In the middle orders the new p stays in shared memory after the
// first pass and the output loop is unrolled by two: unrolled fully with p in
// registers the kernel takes 254 of them, one block a multiprocessor (lx 12, 2.3 M
// points: 119 us, 167 with h2; as separate passes 93 and 106).  With 168 it holds the
// columns; where fewer than three blocks fit so, 128 are better up to lx 12 (77 and
// 84 us there against 94 and 107; lx 11, where three fit, 18 and 23 on 209 thousand
// points), beyond they spill (lx 14, 2.0 M points: 191 us, 127 with 168).  The short
// columns (lx 3, 4) and the long ones that leave one block a multiprocessor either
// way (lx 15, 16) keep p in registers: 421 thousand points at lx 3 16.6 -> 13.5 us,
// 2.5 M at lx 4 49.1 -> 43.3, 2.1 M at lx 16 95.6 -> 97.0, with h2 114.5 -> 98.5.
template <int LX, int NE>
struct AxCgGen {
  static constexpr int L2 = LX * LX, L3 = L2 * LX;
  static constexpr int THREADS = ((L2 * NE + 31) / 32) * 32;
  // p in registers to the end, the output loop unrolled fully
  static constexpr bool HELD = LX == 3 || LX == 4 || LX >= 15;
  static constexpr int UNROLL = HELD ? LX : 2;
  static constexpr int BLOCKS =
      LX == 3 || LX == 4
          ? 0
          : blocks_for(THREADS, LX > 12 || blocks_for(THREADS, 168) >= 3 ? 168 : 128);
  static constexpr size_t SMEM = sizeof(double) * (2 * L2 + (size_t)NE * 3 * L3);
};

template <int LX, int NE, bool H2, typename TZ>
__global__ void __launch_bounds__(AxCgGen<LX, NE>::THREADS, AxCgGen<LX, NE>::BLOCKS)
    ax_cg_gen_kernel(const AxArgs<TZ> a) {
  using C = AxCgGen<LX, NE>;
  constexpr int L2 = C::L2, L3 = C::L3;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double *sD = reinterpret_cast<double *>(smem_raw), *sDt = sD + L2;
  const int tid = threadIdx.x, tz = tid / L2, col = tid - tz * L2;
  const int i = col % LX, j = col / LX;
  double *su = sDt + L2 + (tz < NE ? tz : 0) * 3 * L3, *sur = su + L3, *sus = sur + L3;
  for (int q = tid; q < L2; q += C::THREADS) {
    sD[q] = a.D[q];
    sDt[q] = a.Dt[q];
  }
  chain();
  if (a.st && a.st->done) return;
  const double beta = a.st ? a.st->beta : a.beta;
  double pap = 0.0;
  for (long eb = (long)blockIdx.x * NE; eb < a.nelv; eb += (long)gridDim.x * NE) {
    const long e = eb + tz;
    const bool active = tz < NE && e < a.nelv;
    const long base = e * L3 + col;
    double rp[LX], rut[LX];
    __syncthreads();  // matrices loaded; planes of the previous elements read
    if (active) {
#pragma unroll
      for (int k = 0; k < LX; k++) {
        const long g = base + k * L2;
        rp[k] = (double)a.z[g] + beta * a.p[g];
      }
#pragma unroll
      for (int k = 0; k < LX; k++) {
        a.p[base + k * L2] = rp[k];
        su[col + L2 * k] = rp[k];
      }
    }
    __syncthreads();
    if (active) {
#pragma unroll
      for (int k = 0; k < LX; k++) {
        double ur = 0, us = 0, ut = 0;
#pragma unroll
        for (int l = 0; l < LX; l++) {
          ur += sD[i + LX * l] * su[l + LX * j + L2 * k];
          us += sD[j + LX * l] * su[i + LX * l + L2 * k];
          ut += sD[k + LX * l] * rp[l];
        }
        const long g = base + k * L2;
        const double G11 = __ldg(a.g[0] + g), G22 = __ldg(a.g[1] + g), G33 = __ldg(a.g[2] + g),
                     G12 = __ldg(a.g[3] + g), G13 = __ldg(a.g[4] + g), G23 = __ldg(a.g[5] + g),
                     H = __ldg(a.h1 + g);
        sur[col + L2 * k] = H * (G11 * ur + G12 * us + G13 * ut);
        sus[col + L2 * k] = H * (G12 * ur + G22 * us + G23 * ut);
        rut[k] = H * (G13 * ur + G23 * us + G33 * ut);
      }
    }
    __syncthreads();
    if (active) {
#pragma unroll(C::UNROLL)
      for (int k = 0; k < LX; k++) {
        double c0 = 0, c1 = 0, c2 = 0;
#pragma unroll
        for (int l = 0; l < LX; l++) {
          c0 += sDt[i + LX * l] * sur[l + LX * j + L2 * k];
          c1 += sDt[j + LX * l] * sus[i + LX * l + L2 * k];
          c2 += sDt[k + LX * l] * rut[l];
        }
        const long g = base + k * L2;
        double pk;
        if constexpr (C::HELD)
          pk = rp[k];
        else
          pk = su[col + L2 * k];
        double wv = c0 + c1 + c2;
        if constexpr (H2) wv = wv + __ldg(a.h2 + g) * __ldg(a.B + g) * pk;
        a.w[g] = wv;
        pap += pk * wv;
      }
    }
  }
  double tot;
  if (grid_sum<C::THREADS>(pap, a.partials, a.counter, &tot)) {
    if (a.st) {
      a.st->pap = tot;
      a.st->alpha = a.st->rtz1 / tot;
    } else if (a.pap_out) {
      *a.pap_out = tot;
    }
  }
}

template <int LX, typename TZ>
static cudaError_t launch_ax_cg_gen(const AxArgs<TZ> &a, cudaStream_t s) {
  using C = AxCgGen<LX, AxCfg<LX>::NE>;
  auto kern = a.h2 ? ax_cg_gen_kernel<LX, AxCfg<LX>::NE, true, TZ>
                   : ax_cg_gen_kernel<LX, AxCfg<LX>::NE, false, TZ>;
  if (C::SMEM > 48 * 1024) {
    cudaError_t e =
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
    if (e != cudaSuccess) return e;
  }
  // every partial sum has a slot: blocks loop over the elements beyond that
  const int ne = AxCfg<LX>::NE, need = (a.nelv + ne - 1) / ne;
  launch_chained((long)a.nelv * C::L3, kern,
                 need < a.max_grid ? need : a.max_grid, C::THREADS, C::SMEM, s, a);
  return cudaGetLastError();
}

template <typename TZ>
cudaError_t ax_cg_general(const AxArgs<TZ> &a, int lx, cudaStream_t s) {
  switch (lx) {
#define NB_CG_GEN(N) \
  case N: return launch_ax_cg_gen<N, TZ>(a, s);
    NB_CG_GEN(2) NB_CG_GEN(3) NB_CG_GEN(4) NB_CG_GEN(5) NB_CG_GEN(6) NB_CG_GEN(7) NB_CG_GEN(8)
    NB_CG_GEN(9) NB_CG_GEN(10) NB_CG_GEN(11) NB_CG_GEN(12) NB_CG_GEN(13) NB_CG_GEN(14)
    NB_CG_GEN(15) NB_CG_GEN(16)
#undef NB_CG_GEN
    default: return cudaErrorNotSupported;
  }
}
template cudaError_t ax_cg_general<double>(const AxArgs<double> &, int, cudaStream_t);
template cudaError_t ax_cg_general<float>(const AxArgs<float> &, int, cudaStream_t);

}  // namespace nb
