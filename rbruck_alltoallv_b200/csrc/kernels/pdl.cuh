// Programmatic dependent launch: a kernel launched with launch_dependent() may be scheduled while the kernel before it in
// the stream is still running, as soon as every CTA of that kernel has called pdl_trigger() or left.  It must call
// pdl_wait() before it touches memory: that returns when the kernel before it has completed and its stores are visible.
// Launch latency, barrier set-up and TMEM allocation then overlap with the tail of the previous kernel.  Measured on the
// five to six kernels of a one-rank MoE layer: 176 -> 165 us (fp8, 1024 tokens), 478 -> 474 us (bf16, 64 tokens).
#pragma once
#include <utility>
#include <cuda_runtime.h>

namespace rbv {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... Params, typename... Args>
cudaError_t launch_dependent(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = stream;
  cfg.attrs = &attr; cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

}  // namespace rbv
