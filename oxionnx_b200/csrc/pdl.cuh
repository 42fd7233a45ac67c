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

// Dependent launch only for grids of at most three blocks per SM, where a launch's latency counts.  The blocks of a
// large streaming grid that start beside a tensor-core kernel inherit its split of the SM's memory, nearly all of it
// shared memory, and keep it: with too little L1 for its loads in flight such a grid ran at three quarters of its rate
// (INT8 network at batch 1024: 12.1 -> 12.9 ms).
constexpr unsigned kDependentBlocks = 3 * 148;

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
  cfg.numAttrs = (uint64_t)grid.x * grid.y * grid.z <= kDependentBlocks ? 1 : 0;
  OXB_CUDA(cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(std::forward<Args>(args))...));
}

}  // namespace k
}  // namespace oxb
