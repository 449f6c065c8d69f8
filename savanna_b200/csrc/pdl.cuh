// Kernels that follow each other as programmatic dependents, of two kinds.
//
// In a chain (the Hyena-LI scan, the decode step) a kernel lets the next one start as soon as all its own blocks run, and the next one waits
// for it only when it needs its results.  What does not depend on them - weights, inputs of the whole call - is loaded before the wait, so
// the launch gap and that latency lie behind the kernel before.  The first kernel of a chain is an ordinary launch: it starts after all
// earlier work on the stream, so what the others load ahead is never still being written.
//
// A kernel that is always a dependent (GEMM, attention, its rotary kernel) follows whatever is before it on the stream, which may have let
// it start long before its own end, or may itself be a dependent.  Nothing in global memory is read or written before the wait, weights and
// scalars included: only launch, barriers, tensor memory and descriptors (kernel parameters) are ahead of it.
//
// Every block of a dependent kernel waits before it ends (so kernels end in order) and before its first store.  Results of the kernels
// before must not be read through the non-coherent path, which may hold what was there when the kernel started: no `const __restrict__`
// on pointers to them.
#pragma once
#include <cuda_runtime.h>

namespace sb {

__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// first: an ordinary launch; else a programmatic dependent of the launch before it on the stream (an ordinary one behind anything but a kernel).
template <class... P, class... A>
static int launch_chained(bool first, void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = first ? 0 : 1;
  if (cudaLaunchKernelEx(&cfg, kernel, P(args)...) == cudaSuccess) return 0;
  (void)cudaGetLastError();              // reported here: the next entry point of this thread would take it for its own
  return -2;
}

}  // namespace sb
