// pt2_epi.cu -- k_pt2, plain and batched, for 1 and 2 words per spin string and
// 1, 2, 4 and 8 roots.
#include "pt2_epi.cuh"

namespace cipsi_dev {
template cudaError_t launch_pt2<1, 1, false>(const Params&, const LaunchArgs&, int, cudaStream_t);
template cudaError_t launch_pt2<1, 1, true>(const Params&, const LaunchArgs&, int, cudaStream_t);
template cudaError_t launch_pt2<1, 2, false>(const Params&, const LaunchArgs&, int, cudaStream_t);
template cudaError_t launch_pt2<1, 2, true>(const Params&, const LaunchArgs&, int, cudaStream_t);
template cudaError_t launch_pt2<1, 4, false>(const Params&, const LaunchArgs&, int, cudaStream_t);
template cudaError_t launch_pt2<1, 4, true>(const Params&, const LaunchArgs&, int, cudaStream_t);
template cudaError_t launch_pt2<1, 8, false>(const Params&, const LaunchArgs&, int, cudaStream_t);
template cudaError_t launch_pt2<1, 8, true>(const Params&, const LaunchArgs&, int, cudaStream_t);
template cudaError_t launch_pt2<2, 1, false>(const Params&, const LaunchArgs&, int, cudaStream_t);
template cudaError_t launch_pt2<2, 1, true>(const Params&, const LaunchArgs&, int, cudaStream_t);
template cudaError_t launch_pt2<2, 2, false>(const Params&, const LaunchArgs&, int, cudaStream_t);
template cudaError_t launch_pt2<2, 2, true>(const Params&, const LaunchArgs&, int, cudaStream_t);
template cudaError_t launch_pt2<2, 4, false>(const Params&, const LaunchArgs&, int, cudaStream_t);
template cudaError_t launch_pt2<2, 4, true>(const Params&, const LaunchArgs&, int, cudaStream_t);
template cudaError_t launch_pt2<2, 8, false>(const Params&, const LaunchArgs&, int, cudaStream_t);
template cudaError_t launch_pt2<2, 8, true>(const Params&, const LaunchArgs&, int, cudaStream_t);
}  // namespace cipsi_dev
