// Kernels on the runtime-length block FFT (rp_fft.cuh): contiguous complex signals, columns and rows of the
// four-step transform, axes of multi-dimensional transforms.  H: values a thread holds
// (rp.hpp).  Instantiated by rp_f32.cu, rp_f64.cu, rp_f32_long.cu and rp_f64_long.cu.
#pragma once

#include "launch.hpp"
#include "rp_fft.cuh"

namespace kfr_gpu
{

// four-step twiddle W_N^m = twA[m >> lbits] twB[m & mask]
template <typename T>
__device__ __forceinline__ cpx<T> rp_root(const cpx<T>* __restrict__ A, const cpx<T>* __restrict__ B, long long m,
                                          int lbits)
{
    return ldg(A + (m >> lbits)) * ldg(B + (m & ((1LL << lbits) - 1)));
}

// ---------------------------------------------------------------------------------------------------
// Complex DFT of contiguous signals whose length is a product of primes up to 127: one CTA per tile of
// `spc` signals, the first pass reading and the last pass writing global memory with the lanes along the
// signal (any 8-byte aligned pointers and strides), the CTAs of an SM overlapping one another's accesses.
// Bound by instruction issue (about 25 instructions per element and pass).  4096 signals of 3600 points
// (15 x 16 x 15, one signal per 256-thread CTA): 54 us, 65% of the HBM copy rate (207 us with the
// radix-at-a-time passes before it); 2000 points (four passes) 41%, 100 points (two) 88%.
// ---------------------------------------------------------------------------------------------------
template <typename T, int H>
__global__ void __launch_bounds__(rp_max_threads(2 * sizeof(T), H), 1)
    k_rp_c2c(const __grid_constant__ rp_c2c_args a)
{
    stream_order();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const long long s0 = (long long)blockIdx.x * a.spc;
    const int cnt      = int(a.batch - s0 < a.spc ? a.batch - s0 : a.spc);
    const cpx<T>* in   = reinterpret_cast<const cpx<T>*>(a.in) + s0 * a.istride;
    cpx<T>* out        = reinterpret_cast<cpx<T>*>(a.out) + s0 * a.ostride;
    const bool inv     = a.inverse != 0;
    rp_run<T, H>(
        a.d, reinterpret_cast<cpx<T>*>(smem_raw), cnt, reinterpret_cast<const cpx<T>*>(a.tw),
        [&](int g, int i) { return conj_if(*rp_at(in + g * a.istride, i, uint32_t(sizeof(cpx<T>))), inv); },
        [&](int g, int i, cpx<T> v) { *rp_at(out + g * a.ostride, i, uint32_t(sizeof(cpx<T>))) = conj_if(v, inv); });
}

// ---------------------------------------------------------------------------------------------------
// n-point DFTs down the columns of row-major n x pitch arrays, in the array's own layout: an axis of a
// multi-dimensional transform, or (twiddle) the first pass of a four-step transform of N = n pitch points,
// whose output k of column c is multiplied by W_N^{c k}.  A tile is S columns (128-byte rows where S allows);
// lanes run along the columns, so global and shared accesses are contiguous with no transposition.
// Bound by instruction issue and, for tiles of 4 or 8 columns, by the 32- and 64-byte rows.  Eight 1080 x 1920
// complex arrays, both axes: 150 us; 174 us with the widest tiles that fit one CTA per SM.
// ---------------------------------------------------------------------------------------------------
// RP_AXIS, RP_TABLE: every twiddle from its table.  Powers of two table values (RP_POWERS, RP_MERGE, single precision)
// round more: axes of 1024 to 4096 points 9 to 24% more in all at the same speed, a four-step transform of 2^23 points 30%.
// RP_MERGE: the input is the spectrum X of 2N reals, read as conj(Z[e]) with
//   Z[e] = X[e] + conj X[N-e] + i conj(W_2N^e) (X[e] - conj X[N-e])
// (from_fmt, src/dft/fft-impl.hpp:1852-1896; e = 0 takes the real parts of the first and last bins).  Each bin is
// read by its own column's tile and by the mirrored one, the second time mostly from L2.
enum rp_cols_mode
{
    RP_AXIS,   // no four-step twiddle
    RP_POWERS, // four-step twiddle
    RP_TABLE,
    RP_MERGE
};
template <typename T, int H, rp_cols_mode MODE>
__global__ void __launch_bounds__(rp_max_threads(2 * sizeof(T), H), 1)
    k_rp_cols(const __grid_constant__ rp_strided_args a)
{
    stream_order();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int S       = 1 << a.d.shift;
    const int tiles   = int((a.pitch + S - 1) >> a.d.shift);
    const long long b = blockIdx.x / tiles;
    const int c0      = int(blockIdx.x - b * tiles) << a.d.shift;
    const cpx<T>* in  = reinterpret_cast<const cpx<T>*>(a.in) + b * a.in_stride + c0;
    cpx<T>* out       = reinterpret_cast<cpx<T>*>(a.out) + b * a.out_stride + c0;
    const cpx<T>* twA = reinterpret_cast<const cpx<T>*>(a.twA);
    const cpx<T>* twB = reinterpret_cast<const cpx<T>*>(a.twB);
    // lanes beyond the last column repeat it: they read the same values and store the same results
    const int last  = int(a.pitch - c0 < S ? a.pitch - c0 : S) - 1;
    const bool cin  = a.conj_in != 0, cout = a.conj_out != 0;
    const unsigned long long bytes = a.pitch * sizeof(cpx<T>);
    constexpr bool powers = sizeof(T) == 4 && (MODE == RP_POWERS || MODE == RP_MERGE);
    rp_run<T, H, !powers>(
        a.d, reinterpret_cast<cpx<T>*>(smem_raw), S, reinterpret_cast<const cpx<T>*>(a.tw),
        [&](int g, int i)
        {
            if constexpr (MODE == RP_MERGE)
            {
                const cpx<T>* X   = in - c0;
                const long long N = a.d.n * a.pitch, e = i * a.pitch + c0 + min(g, last);
                if (e == 0)
                {
                    const T x0 = X[0].x, xn = a.ccs ? X[N].x : X[0].y;
                    return mk<T>(x0 + xn, xn - x0);
                }
                const cpx<T> u = X[e], v = conj(X[N - e]);
                const cpx<T> w = ldg(reinterpret_cast<const cpx<T>*>(a.rtw) + e);
                return conj((u + v) + mul_pi(conj(w) * (u - v)));
            }
            else
                return conj_if(*rp_at(in + min(g, last), i, bytes), cin);
        },
        [&](int g, int i, cpx<T> v) { *rp_at(out + min(g, last), i, bytes) = conj_if(v, cout); },
        [&](int g, int k, int step, auto& o)
        {
            if (MODE == RP_AXIS || !twA)
                return;
            constexpr int R     = int(sizeof(o) / sizeof(o[0]));
            const long long col = c0 + min(g, last);
            if constexpr (powers)
            {
                // W^{col k} times powers of the butterfly's step W^{col step}
                if constexpr (R > 4)
                    twiddle_powers4<T, R>(o, rp_root(twA, twB, col * step, a.lbits),
                                          rp_root(twA, twB, 4 * col * step, a.lbits));
                else if constexpr (R > 1)
                    twiddle_powers<T, R>(o, rp_root(twA, twB, col * step, a.lbits));
                const cpx<T> w = rp_root(twA, twB, col * k, a.lbits);
#pragma unroll
                for (int r = 0; r < R; r++)
                    o[r] = o[r] * w;
            }
            else
            {
#pragma unroll
                for (int r = 0; r < R; r++)
                    o[r] = o[r] * rp_root(twA, twB, col * (k + (long long)r * step), a.lbits);
            }
        });
}

// ---------------------------------------------------------------------------------------------------
// Second pass of a four-step transform of N = n1 n points: n-point DFTs along the n1 contiguous rows, output k
// of row k1 to X[k1 + n1 k].  A tile is S rows: the first pass reads along the rows, the others run with the
// lanes across the rows, so the stores cover S consecutive outputs; the transposition is the layout change
// between the first two passes (RP_ROWS).  One complex<double> signal of 2^20 points, both kernels: 181 us,
// 206 us with the radix-at-a-time passes before them (FP64 pipe, latency: one wave of CTAs).
// ---------------------------------------------------------------------------------------------------
template <typename T, int H, bool TABLE>
__global__ void __launch_bounds__(rp_max_threads(2 * sizeof(T), H), 1)
    k_rp_rows(const __grid_constant__ rp_strided_args a)
{
    stream_order();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int S       = 1 << a.d.shift;
    const int tiles   = int((a.pitch + S - 1) >> a.d.shift);
    const long long b = blockIdx.x / tiles;
    const int r0      = int(blockIdx.x - b * tiles) << a.d.shift;
    const int n       = a.d.n;
    const cpx<T>* in  = reinterpret_cast<const cpx<T>*>(a.in) + b * a.in_stride + (long long)r0 * n;
    cpx<T>* out       = reinterpret_cast<cpx<T>*>(a.out) + b * a.out_stride + r0;
    // lanes beyond the last row repeat it
    const int last  = int(a.pitch - r0 < S ? a.pitch - r0 : S) - 1;
    const bool cin  = a.conj_in != 0, cout = a.conj_out != 0;
    const unsigned long long bytes = a.pitch * sizeof(cpx<T>);
    rp_run<T, H, TABLE>(
        a.d, reinterpret_cast<cpx<T>*>(smem_raw), S, reinterpret_cast<const cpx<T>*>(a.tw),
        [&](int g, int i) { return conj_if(*rp_at(in + (long long)min(g, last) * n, i, uint32_t(sizeof(cpx<T>))), cin); },
        [&](int g, int i, cpx<T> v) { *rp_at(out + min(g, last), i, bytes) = conj_if(v, cout); });
}

// ---------------------------------------------------------------------------------------------------
// Second pass of a real forward DFT of 2N reals, N = n1 n: the row DFTs of k_rp_rows, whose outputs Z[k1 + n1 k] stay
// in shared memory, then the split (to_fmt, src/dft/fft-impl.hpp:1799-1841)
//   X[e] = (Z[e] + conj Z[N-e]) / 2 - i W_2N^e (Z[e] - conj Z[N-e]) / 2
// into the spectrum (N + 1 bins, or N packed).  N - e lies in row n1 - k1, so a tile is S / 2 mirror pairs of rows
// (k1, n1 - k1), k1 = 1 .. ; the pair 0 is the rows 0 and n1 / 2, which mirror into themselves.  Two round trips
// instead of three.
// ---------------------------------------------------------------------------------------------------
template <typename T, int H>
__global__ void __launch_bounds__(rp_max_threads(2 * sizeof(T), H), 1)
    k_rp_rows_split(const __grid_constant__ rp_strided_args a)
{
    stream_order();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int S = 1 << a.d.shift, half = S >> 1;
    const int n1 = int(a.pitch), n = a.d.n;
    const int pairs   = (n1 - 1) / 2 + 1;
    const int tiles   = (pairs + half - 1) / half;
    const long long b = blockIdx.x / tiles;
    const int q0      = int(blockIdx.x - b * tiles) * half;
    const long long N = (long long)n1 * n;
    const cpx<T>* in  = reinterpret_cast<const cpx<T>*>(a.in) + b * a.in_stride;
    cpx<T>* out       = reinterpret_cast<cpx<T>*>(a.out) + b * a.out_stride;
    const cpx<T>* rtw = reinterpret_cast<const cpx<T>*>(a.rtw);
    cpx<T>* z         = reinterpret_cast<cpx<T>*>(smem_raw);
    // pair and row of signal g; lanes beyond the last pair repeat it
    const auto pair_of = [&](int g) { return min(q0 + (g & (half - 1)), pairs - 1); };
    const auto row_of  = [&](int g, int q)
    { return g < half ? q : q ? n1 - q : n1 & 1 ? 0 : n1 / 2; };
    rp_run_in<T, H>(a.d, z, S, reinterpret_cast<const cpx<T>*>(a.tw),
                    [&](int g, int i)
                    { return *rp_at(in + (long long)row_of(g, pair_of(g)) * n, i, uint32_t(sizeof(cpx<T>))); });
    for (int i = threadIdx.x; i < S * n; i += blockDim.x)
    {
        const int g = i & (S - 1), k = i >> a.d.shift;
        const int q = pair_of(g), row = row_of(g, q);
        // Z[N - e]: the other row of the pair, or the same row
        const int mg      = q ? g ^ half : g;
        const int mirror  = row ? n - 1 - k : k ? n - k : 0;
        const cpx<T> u    = z[i], v = conj(z[mirror * S + mg]);
        const long long e = row + (long long)n1 * k;
        if (e == 0)
        {
            out[0] = mk<T>(u.x + u.y, a.ccs ? T(0) : u.x - u.y);
            if (a.ccs)
                out[N] = mk<T>(u.x - u.y, T(0));
        }
        else
            out[e] = scale(u + v, T(0.5)) + ldg(rtw + e) * scale(mul_mi(u - v), T(0.5));
    }
}

// ---------------------------------------------------------------------------------------------------

// The four-step passes of k_rp_cols / k_rp_rows for power-of-two lengths known at compile time (C: rp_ct of the pass,
// P: the other length).
template <typename T, class C, int P>
__global__ void __launch_bounds__(C::threads(), 1024 / C::threads()) k_ct_cols(const __grid_constant__ rp_strided_args a)
{
    stream_order();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int S = 1 << C::d.shift, tiles = P / S;
    const long long b = blockIdx.x / tiles;
    const int c0      = int(blockIdx.x % tiles) * S;
    const cpx<T>* in  = reinterpret_cast<const cpx<T>*>(a.in) + b * a.in_stride + c0;
    cpx<T>* out       = reinterpret_cast<cpx<T>*>(a.out) + b * a.out_stride + c0;
    const cpx<T>* twA = reinterpret_cast<const cpx<T>*>(a.twA);
    const cpx<T>* twB = reinterpret_cast<const cpx<T>*>(a.twB);
    const bool cin = a.conj_in != 0;
    rp_run_ct<T, C>(
        reinterpret_cast<cpx<T>*>(smem_raw), reinterpret_cast<const cpx<T>*>(a.tw),
        [&](int g, int i) { return conj_if(in[i * P + g], cin); },
        [&](int g, int i, cpx<T> v) { out[i * P + g] = v; },
        [&](int g, int k, int step, auto& o)
        {
            // W^{col k} times powers of the butterfly's step W^{col step}
            constexpr int R = int(sizeof(o) / sizeof(o[0]));
            const int col   = c0 + g, mask = (1 << a.lbits) - 1;
            const auto root = [&](int m) { return ldg(twA + (m >> a.lbits)) * ldg(twB + (m & mask)); };
            if constexpr (R >= 8)
                twiddle_powers4<T, R>(o, root(col * step), root(4 * col * step));
            else
                twiddle_powers<T, R>(o, root(col * step));
            const cpx<T> w = root(col * k);
#pragma unroll
            for (int r = 0; r < R; r++)
                o[r] = o[r] * w;
        });
}

template <typename T, class C, int P>
__global__ void __launch_bounds__(C::threads(), 1024 / C::threads()) k_ct_rows(const __grid_constant__ rp_strided_args a)
{
    stream_order();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int S = 1 << C::d.shift, tiles = P / S;
    const long long b = blockIdx.x / tiles;
    const int r0      = int(blockIdx.x % tiles) * S;
    const cpx<T>* in  = reinterpret_cast<const cpx<T>*>(a.in) + b * a.in_stride + (long long)r0 * C::d.n;
    cpx<T>* out       = reinterpret_cast<cpx<T>*>(a.out) + b * a.out_stride + r0;
    const bool cout = a.conj_out != 0;
    rp_run_ct<T, C>(
        reinterpret_cast<cpx<T>*>(smem_raw), reinterpret_cast<const cpx<T>*>(a.tw),
        [&](int g, int i) { return in[g * C::d.n + i]; },
        [&](int g, int i, cpx<T> v) { out[i * P + g] = conj_if(v, cout); });
}

template <typename A>
static cudaError_t rp_go(void (*kernel)(const A), const A& a, long long grid, int threads, int smem, cudaStream_t st)
{
    if (grid <= 0)
        return cudaSuccess;
    if (grid > 0x7fffffffLL)
        return cudaErrorInvalidConfiguration;
    if (smem > 48 * 1024)
    {
        const cudaError_t e = prepare_launch(reinterpret_cast<const void*>(kernel), threads, smem);
        if (e != cudaSuccess)
            return e;
    }
    return launch_kernel(kernel, dim3(unsigned(grid)), threads, size_t(smem), st, a);
}

template <typename T, int H>
cudaError_t launch_rp_c2c(const rp_c2c_args& a, int threads, int smem, cudaStream_t st)
{
    return rp_go(k_rp_c2c<T, H>, a, (a.batch + a.spc - 1) / a.spc, threads, smem, st);
}

template <typename T, int H>
cudaError_t launch_rp_strided(const rp_strided_args& a, bool cols, int threads, int smem, cudaStream_t st)
{
    const long long tiles = (a.pitch + (1 << a.d.shift) - 1) >> a.d.shift;
    constexpr bool f64         = sizeof(T) == 8; // always from the tables
    constexpr rp_cols_mode two = f64 ? RP_TABLE : RP_POWERS;
    if (!cols)
        return rp_go(a.table ? k_rp_rows<T, H, true> : k_rp_rows<T, H, f64>, a, tiles * a.batch, threads, smem, st);
    return rp_go(a.rtw     ? k_rp_cols<T, H, RP_MERGE>
                 : !a.twA  ? k_rp_cols<T, H, RP_AXIS>
                 : a.table ? k_rp_cols<T, H, RP_TABLE>
                           : k_rp_cols<T, H, two>,
                 a, tiles * a.batch, threads, smem, st);
}

template <typename T, int H>
cudaError_t launch_rp_rows_split(const rp_strided_args& a, int threads, int smem, cudaStream_t st)
{
    const long long pairs = (a.pitch - 1) / 2 + 1, half = 1LL << (a.d.shift - 1);
    return rp_go(k_rp_rows_split<T, H>, a, (pairs + half - 1) / half * a.batch, threads, smem, st);
}

#define KFR_GPU_RP_INSTANTIATE(T, H)                                                                       \
    template cudaError_t launch_rp_c2c<T, H>(const rp_c2c_args&, int, int, cudaStream_t);                  \
    template cudaError_t launch_rp_strided<T, H>(const rp_strided_args&, bool, int, int, cudaStream_t);    \
    template cudaError_t launch_rp_rows_split<T, H>(const rp_strided_args&, int, int, cudaStream_t);

} // namespace kfr_gpu
