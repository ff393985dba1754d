// nb_precond.h -- Krylov workspace and the preconditioner interface of the
// native solver (the role of pc_t, src/krylov/precon.f90:40-66).
#pragma once

#include <cuda_runtime.h>

#include "nb_gs.h"
#include "nb_nodes.h"
#include "nb_problem.h"

namespace nb {

// Device-resident scalars of one CG solve.
struct CgState {
  double norm_fac, abs_tol;
  double rtz1, rtz2, beta, pap, alpha, rtr, rnorm, res_start;
  int iter, max_iter, done, nan;
  int recompute_every;  // > 0: r = f - A x every that many iterations
  int skip_rc;          // 0 when the current iteration ends with a recompute
  int restart;          // next beta is 0 (after a recompute)
  unsigned long long jump;  // of f, from gs_jump
  // The solve's x and f: the kernels of a captured iteration read them
  // here, so one graph serves every solve of the workspace.
  double *x;
  const double *f;
};

// The iterations form (p, w) of the unassembled w = A p over all local points
// (and the flexible CG its products of an unassembled z), which equals the
// reference's mult-weighted product of the assembled, masked vectors when p is
// continuous and zero on masked points: f then is, and r, z and p with it.  A
// solve whose f is not (its copies differ, or its masked points are not zero, by
// more than kJump of its root mean square: the products then differ by about as
// much) stops before its first iteration with `done` = kRough, and the host goes
// on with iterations that form the reference's products.
constexpr double kJump = 1e-10;
constexpr int kRough = 2;
// st->done of a solve that has not converged at its start
__device__ __forceinline__ int first_done(const CgState *st, long n) {
  return __longlong_as_double((long long)st->jump) > kJump * sqrt(st->rtr / (double)n) ? kRough
                                                                                       : 0;
}

// pc_t%solve(z, r): z = M^-1 r on stream s; returns early when *skip != 0.
struct Precond {
  virtual ~Precond() {}
  virtual cudaError_t apply(double *z, const double *r, const int *skip, cudaStream_t s) = 0;
  // kernels one apply launches
  virtual int launches() const = 0;
  // nonzero when a bounded device wait of an apply expired; clears it
  virtual int take_error() { return 0; }
  // A preconditioner that computes in FP32 may leave its output there: the
  // FP32 array apply_f32 writes (its own buffer), else null.
  virtual const float *output_f32() { return nullptr; }
  virtual cudaError_t apply_f32(const double *r, const int *skip, cudaStream_t s) {
    (void)r;
    (void)skip;
    (void)s;
    return cudaErrorNotSupported;
  }
  // True when apply_dots can form the flexible CG's two inner products
  // (r, mult z) and (w_prev, mult z) of its output: partial sums, two per
  // element, in part; z is written as by apply (or left in FP32 when
  // output_f32 is non-null).
  virtual bool dots_in_apply() const { return false; }
  virtual cudaError_t apply_dots(double *z, const double *r, const double *w_prev, double *part,
                                 const int *skip, cudaStream_t s) {
    (void)z;
    (void)r;
    (void)w_prev;
    (void)part;
    (void)skip;
    (void)s;
    return cudaErrorNotSupported;
  }
};

// Blocks a CG reduction may use (its partial sums live in the workspace).
constexpr int kCgMaxPartials = kMaxRedBlocks;

struct CgWorkspace {
  long n = 0;
  void *base = nullptr;
  size_t bytes = 0;
  double *r = nullptr, *z = nullptr, *p = nullptr, *w = nullptr, *partials = nullptr;
  unsigned *counter = nullptr;
  CgState *st = nullptr;
  void *host_state = nullptr;
  bool use_jacobi = true;
  bool flexible = false;
  bool fused = false;  // the last captured iteration used ax_cg_fused
  bool fold = false;   // z = d r is formed by the x and r update
  int recompute_every = 0;
  // a chunk of iterations, captured: [0] with the local products, [1] with the
  // reference's
  struct Graph {
    cudaGraphExec_t exec = nullptr;
    const void *key[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};
    int launches = 0;
    void drop() {
      if (exec) cudaGraphExecDestroy(exec);
      exec = nullptr;
    }
  } graph[2];
  cudaEvent_t ev = nullptr;  // behind the state copy of the last chunk
  // per-element partial inner products of a preconditioner that forms them
  // (Precond::apply_dots): 2 x nelv doubles, allocated on first use
  double *dots = nullptr;
  long dots_n = 0;
  bool use_dots = false;  // the iterations being captured take them
  ~CgWorkspace();
  cudaError_t ensure(long n);
};

nb_status cg_solve(nb_problem *P, double *x, const double *f, const nb_solve_opts &o,
                   Precond *pc, nb_solve_result *res, cudaStream_t s);

// A CG solve followed without blocking (the batch's concurrent solves).
struct CgRun {
  nb_problem *P = nullptr;
  double *x = nullptr;
  const double *f = nullptr;
  nb_solve_opts o{};
  Precond *pc = nullptr;
  cudaStream_t s = nullptr;
  int chunk = 0, launches = 0;
  bool active = false;
  bool rough = false;  // f is not assembled and masked
};
nb_status cg_start(CgRun &R);
nb_status cg_next_chunk(CgRun &R);
int cg_poll(CgRun &R, bool wait, nb_solve_result *res, nb_status *status);
// Pipelined CG (pipecg.cu).
nb_status pipecg_solve(nb_problem *P, double *x, const double *f, const nb_solve_opts &o,
                       Precond *pc, nb_solve_result *res, cudaStream_t s);
// Restarted flexible GMRES (gmres.cu).
nb_status gmres_solve(nb_problem *P, double *x, const double *f, const nb_solve_opts &o,
                      Precond *pc, nb_solve_result *res, cudaStream_t s);

// Operands of hsmg's coarse level (hsmg_coarse.cu).  T is the precision of
// the middle level; the coarse level is FP64.
template <typename T>
struct CoarseArgs {
  long nelv = 0;
  const T *w_mid = nullptr, *mult_m = nullptr;  // middle-level residual and weights
  const T *J = nullptr;                         // lm x 2 interpolation, column-major
  double *f = nullptr;                          // restricted residual, 8 values an element
};
// blocks of the element-local coarse solve at most (its partial sums)
constexpr int kCoarseMaxBlocks = 1024;

// Vertices up to which the coarse solve works on the assembled matrix: one row
// a thread of the largest cluster (8192; 4096 where the device takes clusters
// of the portable size only).
cudaError_t hsmg_coarse_nodes(int &most);
// The same without any mask.  That problem is singular, and a flexible CG
// carries a change of rounding of its coarse solve into the solution, the more
// the larger the mesh: 1e-14 of it on 12^3 elements, 6e-11 on 16^3, 1e-9 on
// 20^3 and 5e-9 on 32^3 periodic ones, 2e-16 on any with a mask.
constexpr int kCoarseFreeNodes = 4096;
struct CoarseCg {
  NodeOp A;                   // the assembled vertex operator (val null: not built)
  double *f = nullptr;        // element-local right-hand side
  double *x = nullptr;        // solution: a value a node, or 8 an element (val null)
  double norm_fac = 0.0, tol = 0.0;
  int niter = 0, lm = 0, stage_slices = 0;
  int priority = 0;           // of the cluster launch
  const int *skip = nullptr;
  // element-local form
  long nelv = 0;
  double *r = nullptr, *z = nullptr, *p = nullptr, *w = nullptr;
  const double *h1 = nullptr, *g[6] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr},
               *D = nullptr, *Dt = nullptr, *dinv = nullptr, *mult = nullptr;
  double *part = nullptr;   // 2 x 2 x (grid) doubles
  unsigned *bar = nullptr;  // grid-barrier word (reset with err after a timeout)
  int *err = nullptr;       // set to 1 when a barrier wait expired
  GsDevice gs;
};

// f = restriction of (w_mid mult_m), element by element (lm = 3 or 4).
template <typename T>
cudaError_t hsmg_coarse_restrict(const CoarseArgs<T> &a, int lm, const int *skip,
                                 cudaStream_t s, bool chain);
// The coarse Jacobi-CG, one cluster launch.
cudaError_t hsmg_coarse_cg(const CoarseCg &a, const int *skip, cudaStream_t s);

// out = (J x J x J) in from ni to no points an element (down: the transposed
// J), with the transfer kernel of hsmg; cudaErrorNotSupported for pairs it has
// no instantiation of.  J has the larger number of rows.
cudaError_t hsmg_transfer(bool down, int ni, int no, const double *in, const double *J,
                          double *out, long nelv, const int *skip, cudaStream_t s);

// hsmg preconditioner of problem P, built on first use (pc_hsmg.cu).
nb_status hsmg_get(nb_problem *P, const nb_solve_opts &o, Precond **out);

struct PhmgSettings;
// phmg preconditioner of problem P (pc_phmg.cu): the existing one, or one
// built with the defaults; with settings, rebuilt with those.
nb_status phmg_get(nb_problem *P, Precond **out, const PhmgSettings *settings = nullptr);

}  // namespace nb
