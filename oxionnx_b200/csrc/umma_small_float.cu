// Float kinds of the small-problem kernel (see umma_small.cuh); f16 and bf16 are one instantiation.
#include "umma_small.cuh"

namespace oxb {
namespace k {
namespace umma {

void launch_small_tf32(const SmallGroup& g, int grid, size_t smem, int device, cudaStream_t s) { launch_small_kind<KIND_TF32>(g, grid, smem, device, s); }
void launch_small_f16(const SmallGroup& g, int grid, size_t smem, int device, cudaStream_t s) { launch_small_kind<KIND_F16>(g, grid, smem, device, s); }

}  // namespace umma
}  // namespace k
}  // namespace oxb
