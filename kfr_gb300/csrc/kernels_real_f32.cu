// Single-precision real DFT kernels.
#include "kernels.cuh"

namespace kfr_gpu
{
KFR_GPU_INSTANTIATE_REAL(float)
} // namespace kfr_gpu
