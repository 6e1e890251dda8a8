// Four-step passes of the square splits with compile-time indices (KFR_CT_SQUARE_F32).
#include "rp_kernels.cuh"

namespace kfr_gpu
{

bool ct_square_f32(long long n, std::vector<int>& radices)
{
#define KFR_GPU_SQUARE_OF(N, S, ...)                                                                       \
    if (n == N)                                                                                            \
    {                                                                                                      \
        radices = { __VA_ARGS__ };                                                                         \
        return true;                                                                                       \
    }
    KFR_CT_SQUARE_F32(KFR_GPU_SQUARE_OF)
#undef KFR_GPU_SQUARE_OF
    return false;
}

cudaError_t launch_ct_square_f32(const rp_strided_args& a, bool cols, cudaStream_t st)
{
    switch (a.pitch)
    {
#define KFR_GPU_SQUARE_CASE(N, S, ...)                                                                     \
    case N:                                                                                                \
    {                                                                                                      \
        using C = rp_ct<RP_COLS, S, S, __VA_ARGS__>;                                                       \
        using R = rp_ct<RP_ROWS, S, 1, __VA_ARGS__>;                                                       \
        return cols ? rp_go(k_ct_cols<float, C, N>, a, N / S * a.batch, C::threads(), C::d.elems * 8, st)  \
                    : rp_go(k_ct_rows<float, R, N>, a, N / S * a.batch, R::threads(), R::d.elems * 8, st); \
    }
        KFR_CT_SQUARE_F32(KFR_GPU_SQUARE_CASE)
#undef KFR_GPU_SQUARE_CASE
    default: return cudaErrorInvalidValue;
    }
}

} // namespace kfr_gpu
