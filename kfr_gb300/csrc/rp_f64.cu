// Double-precision kernels on the runtime-length block FFT.
#include "rp_kernels.cuh"

namespace kfr_gpu
{
KFR_GPU_RP_INSTANTIATE(double, kRpHold)
} // namespace kfr_gpu
