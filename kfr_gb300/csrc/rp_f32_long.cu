// Single-precision kernels on the runtime-length block FFT, for lengths of more than 16 values per thread.
#include "rp_kernels.cuh"

namespace kfr_gpu
{
KFR_GPU_RP_INSTANTIATE(float, kRpLongHold)
} // namespace kfr_gpu
