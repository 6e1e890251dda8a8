// Single-precision Bluestein and Rader kernels.
#include "kernels.cuh"

namespace kfr_gpu
{
KFR_GPU_INSTANTIATE_CONVOLVED(float)
} // namespace kfr_gpu
