// pt2_w1.cu -- k_cand for one 64-bit word per spin string (norb <= 64),
// plain and batched, for 1, 2, 4 and 8 roots.
#include "pt2_fwd.cuh"

namespace cipsi_dev {
template cudaError_t launch_cand<1, 1, false>(const Params&, const LaunchArgs&, int, cudaStream_t);
template cudaError_t launch_cand<1, 1, true>(const Params&, const LaunchArgs&, int, cudaStream_t);
template cudaError_t launch_cand<1, 2, false>(const Params&, const LaunchArgs&, int, cudaStream_t);
template cudaError_t launch_cand<1, 2, true>(const Params&, const LaunchArgs&, int, cudaStream_t);
template cudaError_t launch_cand<1, 4, false>(const Params&, const LaunchArgs&, int, cudaStream_t);
template cudaError_t launch_cand<1, 4, true>(const Params&, const LaunchArgs&, int, cudaStream_t);
template cudaError_t launch_cand<1, 8, false>(const Params&, const LaunchArgs&, int, cudaStream_t);
template cudaError_t launch_cand<1, 8, true>(const Params&, const LaunchArgs&, int, cudaStream_t);
template int cand_ctas<1, 1>();
template int cand_ctas<1, 2>();
template int cand_ctas<1, 4>();
template int cand_ctas<1, 8>();
}  // namespace cipsi_dev
