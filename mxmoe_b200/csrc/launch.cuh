// Launches whose set-up overlaps the end of the kernel before them in the stream (programmatic dependent launch).
//
// The kernels of a layer form a chain, each reading what the one before wrote.  With a plain launch the next kernel's
// blocks are scheduled only after the last block of the previous one has ended and its writes are flushed.  Launched
// through launch_dependent, a kernel's blocks become resident as soon as every block of the previous kernel has released
// it or ended (and SM resources allow), set up what depends on no earlier kernel and wait in grid_dependency_wait() for the
// previous kernel to have completed with its writes visible.
//
// Rules that every kernel launched this way keeps:
//   * all threads call grid_dependency_wait() before the first access to memory that any kernel reads or writes (only
//     the status block of a problem list, which a copy wrote before the chain began, is read earlier).  A kernel
//     therefore ends after all of its predecessors, and whatever follows it in the stream in the ordinary way does too.
//   * What a kernel of the chain writes is read with ordinary loads: no __ldg, no `const T* __restrict__` parameter.  Both
//     promise data that stays constant for the whole life of the reading kernel; its blocks are resident while their
//     predecessor still writes, and such loads may be moved above the wait.  Weights, their scales, sign vectors, Hadamard
//     factors and problem lists are constant and may be read that way.
//   * release_dependents() comes first: it only lets the next kernel's blocks become resident, and since that happens
//     when the LAST block has called it, no waiting block takes the place of one that still has to start.  Launches of ONE
//     block release early (the routing of a decode batch, the quantisers and the combine of a few tokens): the next
//     kernel's blocks set up on the SMs that stay idle.  Larger launches release when they end: blocks that wait beside
//     running ones cost more than their set-up takes.  Graphs and eager steps, us, everyone releases early / one block
//     only / nobody / plain launches: 500 tokens behind the gate 168.4 / 155.0 / 155.6 / 178.8, 1009 tokens fp16 251.3 /
//     246.7 / 246.3 / 261.7, 61 tokens mixed 142.7 / 138.8 / 138.9 / 140.5, 16 tokens of the mixtral shape 200.5 / 198.0 /
//     197.8 / 198.3, 1 token 63.6 / 63.6 / 65.5 / 64.7, 32 tokens 161.5 / 160.5 / 160.4 / 161.9, 8192 tokens w4a4 429.2 / 431.1 /
//     430.6 / 431.4 (limits of 8 and 32 blocks: 61 tokens mixed 140.0 and 140.1).  The grouped GEMM fills every SM and
//     never releases early.
#pragma once
#include <cuda_runtime.h>

namespace mxb {

__device__ __forceinline__ void release_dependents() {
  if (gridDim.x == 1) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... P, typename... A>
cudaError_t launch_dependent(void (*kernel)(P...), int grid, int threads, size_t smem, cudaStream_t stream, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim            = dim3((unsigned)grid, 1, 1);
  cfg.blockDim           = dim3((unsigned)threads, 1, 1);
  cfg.dynamicSmemBytes   = smem;
  cfg.stream             = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs    = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
  if (e != cudaSuccess) cudaGetLastError();   // the caller reports e; a later launch's check must not find it again
  return e;
}

}  // namespace mxb
