// Programmatic dependent launch for the ordinary kernels: every grid may be scheduled while its predecessor in the
// stream drains, and lets its own successor do the same.
#pragma once

#include <utility>

#include "common.hpp"

namespace oxb {
namespace k {

// First statement of a kernel launched with `launch`: the successor may set itself up from here on (a tensor-core
// kernel has about a microsecond of barriers, tensor memory, weight loads and instruction misses to get out of the
// way), and nothing is read or written before the predecessor's results are visible.
__device__ __forceinline__ void pdl_enter() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <typename... Params, typename... Args>
inline void launch(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  OXB_CUDA(cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(std::forward<Args>(args))...));
}

}  // namespace k
}  // namespace oxb
