// nb_chain.cuh -- launches that chain through programmatic dependent launch.
//
// An operator application, a preconditioner application and the start of a solve
// are chains of kernels of a few microseconds each, and between two of them an
// ordinary stream dependency costs the drain of the first and the launch of the
// second.  A chained kernel lets its successor be scheduled as soon as all of its
// own blocks run (chain_next) and waits for its predecessor's completion and
// memory before it touches anything (chain_wait), so the successor's launch and
// start-up run under the predecessor.
//
// The rules: a kernel launched with the attribute (launch_chained,
// cluster_config) waits before it touches anything that a kernel of the stream
// writes; ahead of the wait it reads index maps and derivative matrices only.  A
// kernel lets its successor go only after its own wait, so a kernel completes
// only after everything before it has, and its successor's wait covers that too.
// A predecessor that does neither (a caller's kernel, the iterations of a solver,
// which run captured) lets its successor go when it completes; a successor
// without the attribute waits for the whole of its predecessor.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace nb {

__device__ __forceinline__ void chain_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void chain_next() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void chain() {
  chain_wait();
  chain_next();
}

// Launches of more points than this are not chained: blocks of the successor
// that wait on a multiprocessor cost a long kernel more than the launch gap.
// Chained at every size, a coupled solve on 3 x 2.1 M points went from 32.1 to
// 36.8 ms and a mixed hsmg solve on 4.1 M from 9.0 to 10.0 ms; the operator on
// 262 thousand points went from 16.5 to 12.5 us, an hsmg application from 70.5 to 65
// us there and from 94 to 90 on 885 thousand (113 and 112 us on 1.4 M: nothing left
// to gain).
constexpr long kChainPoints = 1L << 20;
// Points of a launch that is not chained whatever its size: in an hsmg application
// whose coarse solve is a grid on every multiprocessor, waiting blocks keep that
// grid and the fine level's smoother from their places (lx 4, 28^3 elements, FP32
// smoothing: 383 us chained, 325 not; 346 before there were chained launches).
constexpr long kNotChained = kChainPoints + 1;

// Nor are launches that a graph captures: between the nodes of a graph the gap
// is short already, and waiting blocks cost more than it (Jacobi-CG on 729
// thousand points at lx 10: 18.7 ms chained, 17.0 not).
inline bool chained(long points, cudaStream_t s) {
  if (points > kChainPoints) return false;
  if (!s) return true;  // the legacy stream is never captured
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  return cudaStreamIsCapturing(s, &st) == cudaSuccess && st == cudaStreamCaptureStatusNone;
}

template <typename... P, typename... A>
inline cudaError_t launch_chained(long points, void (*kern)(P...), dim3 grid, dim3 block,
                                  size_t smem, cudaStream_t s, A &&...args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = chained(points, s) ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...);
}

}  // namespace nb
