// pdl.cuh -- programmatic dependent launches of the block LU's kernels.
//
// The factorisation and the solves are chains of hundreds of kernels of a few
// microseconds.  Each of them is launched so that it may start while its
// predecessor in the stream still runs: it sets itself up (barriers, tensor
// memory, tensor maps), then pdl_wait waits until the predecessor has finished
// and its writes are visible, before the first access to memory that any
// other kernel reads or writes; pdl_next then lets its own successor start.  A
// successor is let in only by kernels whose every block is already running,
// so it never keeps a block that it waits for off the SMs.  At 5,400 panels
// (about 1,250 launches per frequency) a mixed frequency takes 23.5 instead of
// 25.5 ms; with eight frequencies in flight the throughput is the same.
#pragma once
#include <cuda_runtime.h>

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <class... P, class... A>
inline cudaError_t pdl_launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
