// Double-precision real DFT kernels.
#include "kernels.cuh"

namespace kfr_gpu
{
KFR_GPU_INSTANTIATE_REAL(double)
} // namespace kfr_gpu
