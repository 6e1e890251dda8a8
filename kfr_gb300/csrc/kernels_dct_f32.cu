// Single-precision DCT kernels.
#include "kernels.cuh"

namespace kfr_gpu
{
KFR_GPU_INSTANTIATE_DCT(float)
} // namespace kfr_gpu
