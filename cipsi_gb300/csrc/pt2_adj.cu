// pt2_adj.cu -- the adjoint form of k_pt2_one (dE2/d integrals and root
// energies), plain form, one 64-bit word per spin string, 1..8 roots
// (pt2_adj_w2.cu: two words).
#include "pt2_kernel.cuh"

namespace cipsi_dev {
template cudaError_t launch_pt2_one<1, 1, true>(const Params&, int, size_t, cudaStream_t);
template cudaError_t launch_pt2_one<1, 2, true>(const Params&, int, size_t, cudaStream_t);
template cudaError_t launch_pt2_one<1, 4, true>(const Params&, int, size_t, cudaStream_t);
template cudaError_t launch_pt2_one<1, 8, true>(const Params&, int, size_t, cudaStream_t);
}  // namespace cipsi_dev
