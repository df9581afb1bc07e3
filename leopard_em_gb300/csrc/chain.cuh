// Kernels of one batch launched as a chain: each is given the programmatic
// launch attribute and waits for its predecessor before it touches memory that
// another kernel wrote or reads.  Its CTAs come in when the predecessor's last
// CTA leaves, without the completion and launch latency in between, and compute
// their root tables meanwhile.
//
// What it is for: batches whose kernels take a few microseconds each.  One
// particle refined: 363 -> 329 us; 24 orientations of 512 x 512: 336 -> 311;
// 1,908: 4.44 -> 4.29 ms; stacks of 1 to 16 crops: 74 -> 65 us.  Letting the
// successor in as soon as the last CTA of a grid has started (an explicit
// trigger) made them slower: its CTAs take slots, shared memory and issue slots
// that the running ones still use (1,908 orientations of 512 x 512 4.46 -> 5.15 ms).
//
// Order: a grid completes only when all its CTAs have waited, so a finished
// predecessor means that everything before it is finished too.  chain_wait()
// therefore comes before any early return, and a kernel launched the plain way
// may stand anywhere between.
#pragma once

#include "common.cuh"

namespace lgb {

__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// After chain_wait(), for each __restrict__ pointer, read or written: the compiler
// need not order accesses through one against an asm that has not seen it, and
// read-only loads carry no order of their own; both could move above the wait.
// (Through the global address, or the compiler would no longer know the address
// space.)
template <class T>
__device__ __forceinline__ T* chain_pointer(T* p) {
  size_t g = __cvta_generic_to_global(p);
  asm volatile("" : "+l"(g)::"memory");
  return static_cast<T*>(__cvta_global_to_generic(g));
}
#define LGB_CHAIN_POINTER(p) p = chain_pointer(p)

template <class... P, class... A>
inline int launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args) {
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...) == cudaSuccess) return LGB_OK;
  cudaGetLastError();
  return LGB_ERR_CUDA;
}

}  // namespace lgb
