// Double-precision DCT kernels.
#include "kernels.cuh"

namespace kfr_gpu
{
KFR_GPU_INSTANTIATE_DCT(double)
} // namespace kfr_gpu
