// Integer kind of the small-problem kernel (see umma_small.cuh).
#include "umma_small.cuh"

namespace oxb {
namespace k {
namespace umma {

void launch_small_i8(const SmallGroup& g, int grid, size_t smem, int device, cudaStream_t s) { launch_small_kind<KIND_I8>(g, grid, smem, device, s); }

}  // namespace umma
}  // namespace k
}  // namespace oxb
