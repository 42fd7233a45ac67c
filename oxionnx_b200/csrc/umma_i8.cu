// Dispatch of the tcgen05 implicit-GEMM kernel for kind::i8; umma_i8_tile.cu holds the instantiations, one object each.
#include "umma_launch.cuh"

namespace oxb {
namespace k {
namespace umma {

extern template void launch_one<32, KIND_I8, false>(const KParams&, int, size_t, int, cudaStream_t);
extern template void launch_one<64, KIND_I8, false>(const KParams&, int, size_t, int, cudaStream_t);
extern template void launch_one<128, KIND_I8, false>(const KParams&, int, size_t, int, cudaStream_t);
extern template void launch_one<256, KIND_I8, false>(const KParams&, int, size_t, int, cudaStream_t);
extern template void launch_one<256, KIND_I8, true>(const KParams&, int, size_t, int, cudaStream_t);
extern template int max_clusters_one<256, KIND_I8, true>(size_t, int);

void launch_kind_i8(const KParams& kp, int bn, bool pair, int grid, size_t smem, int device, cudaStream_t s) {
  launch_any<KIND_I8>(kp, bn, pair, grid, smem, device, s);
}
int max_pairs_kind_i8(size_t smem, int device) { return max_pairs_any<KIND_I8>(smem, device); }

}  // namespace umma
}  // namespace k
}  // namespace oxb
