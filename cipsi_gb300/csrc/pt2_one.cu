// pt2_one.cu -- the forward form of k_pt2_one (runs in the memory of the
// neighbour lists alone), one and two 64-bit words per spin string, 1..8 roots.
#include "pt2_kernel.cuh"

namespace cipsi_dev {
template cudaError_t launch_pt2_one<1, 1, false>(const Params&, int, size_t, cudaStream_t);
template cudaError_t launch_pt2_one<1, 2, false>(const Params&, int, size_t, cudaStream_t);
template cudaError_t launch_pt2_one<1, 4, false>(const Params&, int, size_t, cudaStream_t);
template cudaError_t launch_pt2_one<1, 8, false>(const Params&, int, size_t, cudaStream_t);
template cudaError_t launch_pt2_one<2, 1, false>(const Params&, int, size_t, cudaStream_t);
template cudaError_t launch_pt2_one<2, 2, false>(const Params&, int, size_t, cudaStream_t);
template cudaError_t launch_pt2_one<2, 4, false>(const Params&, int, size_t, cudaStream_t);
template cudaError_t launch_pt2_one<2, 8, false>(const Params&, int, size_t, cudaStream_t);
}  // namespace cipsi_dev
