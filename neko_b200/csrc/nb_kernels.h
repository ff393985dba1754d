// nb_kernels.h -- launchers shared between the CUDA translation units.
#pragma once

#include <cuda_runtime.h>

#include "nb_internal.h"

namespace nb {

// Stream used by drop-in entry points that take none: the one set by
// nb_set_default_stream, else Neko's glb_cmd_queue when the program defines
// it, else the legacy default stream.
cudaStream_t default_stream();
void set_default_stream(cudaStream_t s);

// w = A u (+ h2 B u when h2 is given), any lx in 2..16.
template <typename T>
cudaError_t ax_helm(T *w, const T *u, const T *dx, const T *dy, const T *dz, const T *dxt,
                    const T *dyt, const T *dzt, const T *h1, const T *g11, const T *g22,
                    const T *g33, const T *g12, const T *g13, const T *g23, int nelv, int lx,
                    cudaStream_t s, const int *skip = nullptr, const T *h2 = nullptr,
                    const T *B = nullptr);

// Persistent bulk-copy variant of ax_helm (dx = dy = dz) for lx 4..10; returns
// cudaErrorNotSupported for other lx and when the pointers are not 16-byte
// aligned.
cudaError_t ax_helm_stream(double *w, const double *u, const double *D, const double *Dt,
                           const double *h1, const double *g11, const double *g22,
                           const double *g33, const double *g12, const double *g13,
                           const double *g23, const double *h2, const double *B, int nelv, int lx,
                           cudaStream_t s, const int *skip = nullptr, int *err = nullptr);

// True when dx, dy, dz (and dxt, dyt, dzt) hold the same lx x lx matrix
// (pointer-equal, or equal contents, compared once per pointer set).
bool same_derivatives(const void *dx, const void *dy, const void *dz, const void *dxt,
                      const void *dyt, const void *dzt, int lx);

// Reads and clears the error word of the drop-in cuda_ax_helm (0 = no
// error); kernels given a null error word record their timeouts there.
int take_dropin_error();
// Device address of that word on the current device (looked up once).
int *dropin_error_word();

// (au, av, aw) = A (u, v, w), one set of coefficients, plus h2 B (u, v, w)
// when h2 is given (ax_vector.cu).
cudaError_t ax_helm_vector(double *au, double *av, double *aw, const double *u,
                           const double *v, const double *w, const double *D,
                           const double *Dt, const double *h1, const double *g11,
                           const double *g22, const double *g33, const double *g12,
                           const double *g13, const double *g23, const double *h2,
                           const double *B, int nelv, int lx, cudaStream_t s, int *err,
                           const int *skip = nullptr);

// (au, av, aw) = A_stress (u, v, w): the full-stress operator with
// cofactors cof[0..8] = drdx, drdy, drdz, dsdx, dsdy, dsdz, dtdx, dtdy, dtdz
// (ax_stress.cu), plus h2 B (u, v, w) when h2 is given (in the same pass on
// the streaming kernel).  Returns at once when *skip is set.
cudaError_t ax_stress(double *au, double *av, double *aw, const double *u, const double *v,
                      const double *w, const double *dx, const double *dy, const double *dz,
                      const double *h1, const double *jacinv, const double *const cof[9],
                      const double *w3, int nelv, int lx, cudaStream_t s, int *err,
                      const int *skip, const double *h2 = nullptr, const double *Bm = nullptr);
// au += h2 B u, av += h2 B v, aw += h2 B w
cudaError_t ax_stress_part2(double *au, double *av, double *aw, const double *u,
                            const double *v, const double *w, const double *h2,
                            const double *B, long n, cudaStream_t s, const int *skip);

struct CgState;
// p = z + beta p, w = A p (+ h2 B p when h2 is given; no gather-scatter) and
// pap = sum p * w in one launch (ax_helm.cu).  With a CG state, beta is read
// from it, the launch returns at once when st->done is set, and pap and
// alpha = rtz / pap are written to it; without one, beta is the argument and
// pap goes to *pap_out (device, may be null).  The streaming kernel for lx 4
// to 10 with 16-byte aligned operands (even lx with an FP32 z), a general one
// otherwise;
// cudaErrorNotSupported for lx outside 2..16.
// z may be FP32 (a mixed-precision preconditioner's output), widened as read.
template <typename TZ>
cudaError_t ax_cg_fused(double *w, double *p, const TZ *z, const double *D, const double *Dt,
                        const double *h1, const double *g11, const double *g22, const double *g33,
                        const double *g12, const double *g13, const double *g23,
                        const double *h2, const double *B, int nelv, int lx, CgState *st,
                        double beta, double *pap_out, double *partials, unsigned *counter,
                        int max_grid, cudaStream_t s, int *err);

// cuda_fdm_do_fast for nl 8..16 with the native FDM passes (pc_hsmg.cu);
// cudaErrorNotSupported for other nl.
cudaError_t fdm_dropin(double *eo, double *r, const double *s, const double *d, int nl, int nel,
                       cudaStream_t st);

// Grid size for streaming kernels: a multiple of the SM count.
int stream_grid(long n, int threads);

}  // namespace nb
