// One tile width of the tcgen05 implicit-GEMM kernel for kind::i8 (OXB_TILE columns, a CTA pair or a lone CTA).
#include "umma_launch.cuh"

namespace oxb {
namespace k {
namespace umma {

template void launch_one<OXB_TILE, KIND_I8, OXB_PAIR>(const KParams&, int, size_t, int, cudaStream_t);
template int max_clusters_one<OXB_TILE, KIND_I8, OXB_PAIR>(size_t, int);

}  // namespace umma
}  // namespace k
}  // namespace oxb
