// pt2_adj_w2.cu -- the adjoint kernel k_pt2_adj, plain form, two 64-bit
// words per spin string (norb 65..128), 1..8 roots; a unit of its own so
// that the build compiles it beside pt2_adj.cu.
#include "pt2_kernel.cuh"

namespace cipsi_dev {
template cudaError_t launch_pt2_adj<2, 1>(const Params&, int, size_t, cudaStream_t);
template cudaError_t launch_pt2_adj<2, 2>(const Params&, int, size_t, cudaStream_t);
template cudaError_t launch_pt2_adj<2, 4>(const Params&, int, size_t, cudaStream_t);
template cudaError_t launch_pt2_adj<2, 8>(const Params&, int, size_t, cudaStream_t);
}  // namespace cipsi_dev
