// pt2_adj.cu -- the adjoint kernel k_pt2_adj (dE2/d integrals and root
// energies), plain form, one 64-bit word per spin string, 1..8 roots
// (pt2_adj_w2.cu: two words).
#include "pt2_kernel.cuh"

namespace cipsi_dev {
template cudaError_t launch_pt2_adj<1, 1>(const Params&, int, size_t, cudaStream_t);
template cudaError_t launch_pt2_adj<1, 2>(const Params&, int, size_t, cudaStream_t);
template cudaError_t launch_pt2_adj<1, 4>(const Params&, int, size_t, cudaStream_t);
template cudaError_t launch_pt2_adj<1, 8>(const Params&, int, size_t, cudaStream_t);
}  // namespace cipsi_dev
