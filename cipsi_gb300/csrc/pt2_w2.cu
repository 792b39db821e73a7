// pt2_w2.cu -- k_cand for two 64-bit words per spin string (norb <= 128),
// plain and batched, for 1, 2, 4 and 8 roots.
#include "pt2_fwd.cuh"

namespace cipsi_dev {
template cudaError_t launch_cand<2, 1, false>(const Params&, const LaunchArgs&, int, cudaStream_t);
template cudaError_t launch_cand<2, 1, true>(const Params&, const LaunchArgs&, int, cudaStream_t);
template cudaError_t launch_cand<2, 2, false>(const Params&, const LaunchArgs&, int, cudaStream_t);
template cudaError_t launch_cand<2, 2, true>(const Params&, const LaunchArgs&, int, cudaStream_t);
template cudaError_t launch_cand<2, 4, false>(const Params&, const LaunchArgs&, int, cudaStream_t);
template cudaError_t launch_cand<2, 4, true>(const Params&, const LaunchArgs&, int, cudaStream_t);
template cudaError_t launch_cand<2, 8, false>(const Params&, const LaunchArgs&, int, cudaStream_t);
template cudaError_t launch_cand<2, 8, true>(const Params&, const LaunchArgs&, int, cudaStream_t);
template int cand_ctas<2, 1>();
template int cand_ctas<2, 2>();
template int cand_ctas<2, 4>();
template int cand_ctas<2, 8>();
}  // namespace cipsi_dev
