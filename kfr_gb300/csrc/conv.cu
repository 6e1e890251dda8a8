// FFT convolution filter kernels and host class (see conv.hpp).
#include "conv.hpp"
#include "conv16.cuh"
#include "convolve.hpp"
#include "kernels.cuh"
#include "rp_fft.cuh"
#include "workspace.hpp"

#include <algorithm>
#include <vector>

namespace kfr_gpu
{

// Real-DFT split of bins (k, c-k) from the c-point complex spectrum of the packed reals.
template <typename T>
__device__ __forceinline__ cpx<T> rsplit(cpx<T> zk, cpx<T> zkk, cpx<T> w)
{
    const cpx<T> znk = conj(zkk);
    return scale(zk + znk, T(0.5)) + w * scale(mul_mi(zk - znk), T(0.5));
}
// Real-DFT merge (inverse of rsplit, times 2) of bins (k, c-k).
template <typename T>
__device__ __forceinline__ cpx<T> rmerge(cpx<T> yk, cpx<T> ykk, cpx<T> w)
{
    const cpx<T> ynk = conj(ykk);
    return (yk + ynk) + mul_pi(conj(w) * (yk - ynk));
}

// Block FFT of one signal per CTA between global memory and one shared buffer, for convolution blocks of any length
// (the runtime-length block FFT, in place):
//   to_smem(ld):   c-point DFT of ld(i), i < c, left at buf[pos(k)]; ends with a barrier;
//   from_smem(st): c-point DFT of buf[pos(i)], output k to st(k, x).
template <typename T>
struct conv_rp
{
    using real                       = T;
    static constexpr int max_threads = rp_max_threads(2 * sizeof(T), kRpHold);
    cpx<T>* buf;
    const cpx<T>* tw;
    const rp_desc& d;
    __device__ __forceinline__ conv_rp(cpx<T>* b, const void* t, const conv_fft& f)
        : buf(b), tw(reinterpret_cast<const cpx<T>*>(t)), d(f.rp)
    {
    }
    __device__ __forceinline__ int n() const { return d.n; }
    static __device__ __forceinline__ int pos(int i) { return i; }
    template <class LD>
    __device__ __forceinline__ void to_smem(const LD& ld) const
    {
        for (int i = threadIdx.x; i < d.n; i += blockDim.x)
            buf[i] = ld(i);
        __syncthreads();
        rp_run_smem<T>(d, buf, 1, tw);
    }
    template <class ST>
    __device__ __forceinline__ void from_smem(const ST& st) const
    {
        rp_run_smem<T>(d, buf, 1, tw);
        for (int k = threadIdx.x; k < d.n; k += blockDim.x)
            st(k, buf[k]);
    }
};

// The same for blocks of F = 2048 and 4096 samples, with a compile-time transform whose twiddles all come from the table
// (conv_rp's powers of two table values round more: 1.34 times the relative RMS error at F = 2048, 1.27 times at 4096).
// 64 channels of 2^20 samples through 513 taps: 373 us with conv_rp from the table, 340 with this one.
template <int N, int TS, int... Rs>
struct conv_ct
{
    using real                       = float;
    static constexpr int max_threads = ct_fft<float, N, TS, Rs...>::max_threads;
    cpx<float>* buf;
    const cpx<float>* tw;
    __device__ __forceinline__ conv_ct(cpx<float>* b, const void* t, const conv_fft&)
        : buf(b), tw(reinterpret_cast<const cpx<float>*>(t))
    {
    }
    static __device__ __forceinline__ int n() { return N; }
    static __device__ __forceinline__ int pos(int i) { return ct_fft<float, N, TS, Rs...>::pi(i); }
    __device__ __forceinline__ void run() const
    {
        // TS threads, all of them with butterflies (the mask tells the compiler: values that look conditional count as
        // live around the loop of k_fir_bwd, which then spills)
        static_assert((TS & (TS - 1)) == 0 && N % (16 * TS) == 0, "whole butterflies per thread");
        cpx<float> v[ct_ept<N, TS, Rs...>()];
        ct_passes<float, N, TS, ct_ept<N, TS, Rs...>(), 1, 0, Rs...>(v, buf, tw, int(threadIdx.x) & (TS - 1));
    }
    template <class LD>
    __device__ __forceinline__ void to_smem(const LD& ld) const
    {
        for (int i = threadIdx.x; i < N; i += blockDim.x)
            buf[pos(i)] = ld(i);
        __syncthreads();
        run();
    }
    template <class ST>
    __device__ __forceinline__ void from_smem(const ST& st) const
    {
        run();
        for (int k = threadIdx.x; k < N; k += blockDim.x)
            st(k, buf[pos(k)]);
    }
};

// GO(P) with the block FFT of f.
#define KFR_GPU_CONV_CT_CASE(N, TS, ...)                                                                   \
    case N: return go(conv_tag<conv_ct<N, TS, __VA_ARGS__>>{});
template <class P>
struct conv_tag
{
    using type = P;
};
template <typename T, class GO>
static auto conv_dispatch(const conv_fft& f, const GO& go)
{
    if constexpr (std::is_same<T, float>::value)
        switch (f.ct)
        {
            KFR_CT_CONV_F32(KFR_GPU_CONV_CT_CASE)
        default: break;
        }
    return go(conv_tag<conv_rp<T>>{});
}
#undef KFR_GPU_CONV_CT_CASE

// Reals (x[i], x[i + 1]) of the n reals at x, zero outside; pairs: even i are 8-byte (16-byte) aligned.
template <typename T>
__device__ __forceinline__ cpx<T> real_pair(const T* x, long long i, long long n, bool pairs)
{
    if (pairs && i >= 0 && i + 1 < n)
        return *reinterpret_cast<const cpx<T>*>(x + i);
    return mk<T>(i >= 0 && i < n ? x[i] : T(0), i + 1 >= 0 && i + 1 < n ? x[i + 1] : T(0));
}
template <typename T>
__device__ __forceinline__ void put_pair(T* y, long long i, long long n, bool pairs, cpx<T> v)
{
    if (pairs && i + 1 < n)
        *reinterpret_cast<cpx<T>*>(y + i) = v;
    else
    {
        if (i < n)
            y[i] = v.x;
        if (i + 1 < n)
            y[i + 1] = v.y;
    }
}
template <typename T>
__device__ __forceinline__ bool pair_aligned(const void* p)
{
    return (reinterpret_cast<uintptr_t>(p) & (2 * sizeof(T) - 1)) == 0;
}

// One overlap-save block per CTA: blockIdx.x = output block, blockIdx.y = channel.  The overlap a.m1 is even (a
// zero tap is added to an even tap count), so blocks start at even samples and move as pairs.
template <class P>
__global__ void __launch_bounds__(P::max_threads, 1)
    k_conv_os(const __grid_constant__ conv_args a)
{
    stream_order();
    using T = typename P::real;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const P fft(reinterpret_cast<cpx<T>*>(smem_raw), a.tw, a.fft);
    cpx<T>* sm = fft.buf;
    const int c           = fft.n();
    const int ch          = blockIdx.y;
    const T* in           = reinterpret_cast<const T*>(a.in) + (long long)ch * a.n;
    const T* hist         = reinterpret_cast<const T*>(a.hist) + (long long)ch * a.nhist;
    T* out                = reinterpret_cast<T*>(a.out) + (long long)ch * a.n;
    const long long start = (long long)blockIdx.x * a.bo - a.m1; // sample of the block's first input
    const bool in_pairs   = pair_aligned<T>(in);
    if (start >= 0 && start + 2 * c <= a.n && in_pairs)
    {
        // inside the input (uniform: one of the two calls runs)
        const T* x = in + start;
        fft.to_smem([x](int m) { return *reinterpret_cast<const cpx<T>*>(x + 2 * m); });
    }
    else
        fft.to_smem(
            [&](int m)
            {
                const long long i = start + 2 * m;
                if (i >= 0)
                    return real_pair<T>(in, i, a.n, in_pairs);
                // samples before the call (i is even), the latest of them at hist[nhist - 1]
                const long long h = i + a.nhist;
                return mk<T>(h >= 0 ? hist[h] : T(0), h + 1 >= 0 ? hist[h + 1] : T(0));
            });
    const cpx<T>* H   = reinterpret_cast<const cpx<T>*>(a.hspec);
    const cpx<T>* rtw = reinterpret_cast<const cpx<T>*>(a.rtw);
    for (int k = threadIdx.x; k <= c / 2; k += blockDim.x)
    {
        if (k == 0)
        {
            const cpx<T> z0 = sm[0];
            const T y0      = (z0.x + z0.y) * ldg(H).x;
            const T yc      = (z0.x - z0.y) * ldg(H + c).x;
            sm[0]           = conj(mk(y0 + yc, y0 - yc));
        }
        else
        {
            const int kk      = c - k;
            const cpx<T> zk   = sm[P::pos(k)];
            const cpx<T> zkk  = sm[P::pos(kk)];
            const cpx<T> wk   = ldg(rtw + k);
            const cpx<T> wkk  = mk<T>(-wk.x, wk.y); // W_F^(c - k) = -conj(W_F^k)
            const cpx<T> yk   = rsplit(zk, zkk, wk) * ldg(H + k);
            const cpx<T> ykk  = rsplit(zkk, zk, wkk) * ldg(H + kk);
            sm[P::pos(k)]     = conj(rmerge(yk, ykk, wk));
            if (kk != k)
                sm[P::pos(kk)] = conj(rmerge(ykk, yk, wkk));
        }
    }
    __syncthreads();
    // output u of the inverse holds samples 2u and 2u + 1 of the block (conjugated); the first a.m1 are the
    // wrapped-around overlap
    const long long first = (long long)blockIdx.x * a.bo;
    const int skip        = int(a.m1 >> 1);
    const bool out_pairs  = pair_aligned<T>(out);
    fft.from_smem(
        [&](int u, cpx<T> v)
        {
            if (u >= skip)
                put_pair<T>(out, first + 2 * (u - skip), a.n, out_pairs, conj(v));
        });
}

// ---------------------------------------------------------------------------------------------------
// Gradients of a causal FIR filter, block by block in the frequency domain.  Block t0 of channel c takes
// F = 2c samples of the output gradient g from t0 and B = F - m1 samples of the input x from t0, zero padded:
//   grad_x[t0 + t] = sum_m h[m] g[t0 + t + m] = IDFT(G conj(H))[t], t < B;
//   grad_h[m]     += sum_t x[t0 + t] g[t0 + t + m] = IDFT(G conj(X))[m], m <= m1 (no wrap-around),
// so both share G, and the second sum stays a spectrum until all blocks are added.  Persistent CTAs, each with
// its own sum in shared memory (every bin owned by one thread); k_fir_reduce adds them in a fixed order and
// k_fir_taps_inner and _outer transform the sum back.  Bound by instruction issue (three c-point FFTs per block).  64 channels
// of 2^20 samples, 1023 taps, forward and both gradients: 6397 -> 869 us against reversed copies through the
// filter and real DFTs of 2^21 points per channel; 664 us with the paired blocks below.
// ---------------------------------------------------------------------------------------------------
template <class P>
__global__ void __launch_bounds__(P::max_threads, 1)
    k_fir_bwd(const __grid_constant__ fir_bwd_args a)
{
    stream_order();
    using T = typename P::real;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const P fg(reinterpret_cast<cpx<T>*>(smem_raw), a.tw, a.fft);
    const P fx(fg.buf + a.elems, a.tw, a.fft);
    cpx<T>* sg        = fg.buf;
    cpx<T>* sx        = fx.buf;
    cpx<T>* acc       = sx + a.elems;
    const int c       = fg.n();
    const cpx<T>* H   = reinterpret_cast<const cpx<T>*>(a.hspec);
    const cpx<T>* rtw = reinterpret_cast<const cpx<T>*>(a.rtw);
    const bool want_x = a.grad_x != nullptr, want_h = a.partial != nullptr;
    if (want_h)
        for (int k = threadIdx.x; k <= c / 2; k += blockDim.x)
            acc[k] = acc[c - k] = mk<T>(0, 0);
    for (long long b = blockIdx.x; b < a.blocks * a.channels; b += gridDim.x)
    {
        const long long ch = b / a.blocks, t0 = (b - ch * a.blocks) * a.bo;
        const T* g = reinterpret_cast<const T*>(a.grad_y) + ch * a.n;
        const T* x = reinterpret_cast<const T*>(a.x) + ch * a.n;
        const bool gp = pair_aligned<T>(g), xp = pair_aligned<T>(x);
        if (t0 + 2 * c <= a.n && gp)
        {
            const T* gt = g + t0;
            fg.to_smem([gt](int m) { return *reinterpret_cast<const cpx<T>*>(gt + 2 * m); });
        }
        else
            fg.to_smem([&](int m) { return real_pair<T>(g, t0 + 2 * m, a.n, gp); });
        if (want_h)
        {
            const long long xn = t0 + a.bo < a.n ? t0 + a.bo : a.n; // a.bo is even
            fx.to_smem([&](int m) { return real_pair<T>(x, t0 + 2 * m, xn, xp); });
        }
        for (int k = threadIdx.x; k <= c / 2; k += blockDim.x)
        {
            if (k == 0)
            {
                const cpx<T> zg = sg[0];
                const T g0 = zg.x + zg.y, gc = zg.x - zg.y;
                if (want_h)
                {
                    const cpx<T> zx = sx[0];
                    acc[0].x += g0 * (zx.x + zx.y);
                    acc[c].x += gc * (zx.x - zx.y);
                }
                if (want_x)
                {
                    const T y0 = g0 * ldg(H).x, yc = gc * ldg(H + c).x;
                    sg[0]      = conj(mk(y0 + yc, y0 - yc));
                }
            }
            else
            {
                const int kk     = c - k;
                const cpx<T> wk  = ldg(rtw + k);
                const cpx<T> wkk = mk<T>(-wk.x, wk.y); // W_F^(c - k) = -conj(W_F^k)
                const cpx<T> zk = sg[P::pos(k)], zkk = sg[P::pos(kk)];
                const cpx<T> gk = rsplit(zk, zkk, wk), gkk = rsplit(zkk, zk, wkk);
                if (want_h)
                {
                    const cpx<T> uk = sx[P::pos(k)], ukk = sx[P::pos(kk)];
                    acc[k] = acc[k] + gk * conj(rsplit(uk, ukk, wk));
                    if (kk != k)
                        acc[kk] = acc[kk] + gkk * conj(rsplit(ukk, uk, wkk));
                }
                if (want_x)
                {
                    const cpx<T> yk = gk * conj(ldg(H + k)), ykk = gkk * conj(ldg(H + kk));
                    sg[P::pos(k)] = conj(rmerge(yk, ykk, wk));
                    if (kk != k)
                        sg[P::pos(kk)] = conj(rmerge(ykk, yk, wkk));
                }
            }
        }
        __syncthreads();
        if (want_x)
        {
            T* gx              = reinterpret_cast<T*>(a.grad_x) + ch * a.n;
            const long long xn = t0 + a.bo < a.n ? t0 + a.bo : a.n;
            const bool op      = pair_aligned<T>(gx);
            fg.from_smem(
                [&](int u, cpx<T> v)
                {
                    if (2 * u < a.bo)
                        put_pair<T>(gx, t0 + 2 * u, xn, op, conj(v));
                });
            __syncthreads();
        }
    }
    if (want_h)
    {
        cpx<T>* p = reinterpret_cast<cpx<T>*>(a.partial) + (long long)blockIdx.x * (c + 1);
        for (int k = threadIdx.x; k <= c / 2; k += blockDim.x)
        {
            p[k] = acc[k];
            if (c - k != k)
                p[c - k] = acc[c - k];
        }
    }
}

// sum[k] = sum over `parts` partial spectra of `bins` values: 32 bins per CTA, 8 rows of threads over the parts.
template <typename T>
__global__ void __launch_bounds__(256) k_fir_reduce(cpx<T>* sum, const cpx<T>* partial, int parts, int bins)
{
    stream_order();
    __shared__ cpx<T> s[8][32];
    const int k = blockIdx.x * 32 + int(threadIdx.x & 31), row = threadIdx.x >> 5;
    cpx<T> v = mk<T>(0, 0);
    if (k < bins)
        for (int p = row; p < parts; p += 8)
            v = v + partial[(long long)p * bins + k];
    s[row][threadIdx.x & 31] = v;
    __syncthreads();
    if (row == 0 && k < bins)
    {
        for (int r = 1; r < 8; r++)
            v = v + s[r][threadIdx.x & 31];
        sum[k] = v;
    }
}

// Spectrum of the taps, H[k] = sum_m h[m] W_F^{m k} / F for k <= c, in double precision on the device, as sums
// over m = m1 Q + m0: first the inner sums S[m0][k mod F/Q] = sum_{m1} h[m1 Q + m0] W_F^{Q m1 k}, then
// H[k] = sum_{m0} W_F^{m0 k} S[m0][k mod F/Q].  w: W_F^j, j < F; placed: stored for k_fir16_bwd.  (FP64 FFTs of one CTA
// would take tens of microseconds on this part; these sums spread over all SMs.)
template <typename T>
__global__ void __launch_bounds__(128) k_fir_spec_inner(double2* S, const T* h, const double2* __restrict__ w,
                                                       int taps, int F, int Q)
{
    stream_order();
    const int P = F / Q, i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= Q * P)
        return;
    const int m0 = i / P, k = i - m0 * P;
    double re = 0, im = 0;
    int at = 0; // (Q m1 k) mod F
    for (int m = m0; m < taps; m += Q)
    {
        const double v = double(h[m]);
        const double2 r = w[at];
        re += v * r.x;
        im += v * r.y;
        at += Q * k;
        if (at >= F)
            at -= F;
    }
    S[i] = make_double2(re, im);
}
// The sum over the four lanes that share an output.  (A warp's FP64 instruction takes 64 cycles of one of the SM's four
// schedulers, so the sums below are dealt to four times as many warps: 600 taps, k_fir_spec_outer 28.5 -> 12.8 us.)
__device__ __forceinline__ double sum_of_4(double v)
{
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    return v + __shfl_xor_sync(0xffffffffu, v, 2);
}
template <typename T>
__global__ void __launch_bounds__(128) k_fir_spec_outer(cpx<T>* H, const double2* __restrict__ S,
                                                       const double2* __restrict__ w, int taps, int F, int Q,
                                                       bool placed)
{
    stream_order();
    const int i = blockIdx.x * blockDim.x + threadIdx.x, part = i & 3;
    const int k = min(i >> 2, F / 2); // lanes past the last bin repeat it
    const int P = F / Q, kp = k & (P - 1), rows = taps < Q ? taps : Q;
    double re = 0, im = 0;
#pragma unroll 4
    for (int m0 = part; m0 < rows; m0 += 4)
    {
        const double2 s = __ldg(S + m0 * P + kp), r = __ldg(w + (m0 * k & (F - 1)));
        re += s.x * r.x - s.y * r.y;
        im += s.x * r.y + s.y * r.x;
    }
    re = sum_of_4(re);
    im = sum_of_4(im);
    if (part)
        return;
    const cpx<T> h = mk<T>(T(re / F), T(im / F));
    if (!placed)
        H[k] = h;
    else
    {
        // all F bins in fft16_place order
        H[fft16_place(k)]           = h;
        H[fft16_place((F - k) % F)] = conj(h);
    }
}

// Taps gradient from the summed spectrum, grad_h[m] = Re sum_k S[k] W_F^{-m k} / F for m < taps, in double precision as the
// taps' spectrum above: inner sums U[k0][m mod P] over k = k1 Q + k0, P = F / Q, then the sum over k0.  placed: all F bins
// in fft16_place order; otherwise the bins k <= F / 2 of a Hermitian spectrum.  In single precision this last transform
// alone made up a third of the gradient's squared rounding error (one channel of 4096 samples, 16 to 300 taps: 1.2 times
// the error of whole-signal transforms, in double precision the same).
template <typename T>
__global__ void __launch_bounds__(128) k_fir_taps_inner(double2* U, const cpx<T>* __restrict__ S,
                                                       const double2* __restrict__ w, int F, int Q, bool placed)
{
    stream_order();
    const int t = blockIdx.x * blockDim.x + threadIdx.x, part = t & 3;
    const int P = F / Q, i = min(t >> 2, F - 1), k0 = i / P, m = i - k0 * P;
    double re = 0, im = 0;
#pragma unroll 4
    for (int k1 = part; k1 < P; k1 += 4)
    {
        const int k     = k1 * Q + k0;
        const bool up   = placed || k <= F / 2;
        const cpx<T> s  = ldg(S + (placed ? fft16_place(k) : up ? k : F - k));
        const double x = double(s.x), y = up ? double(s.y) : -double(s.y);
        const double2 r = __ldg(w + (Q * k1 * m & (F - 1)));
        re += x * r.x + y * r.y;
        im += y * r.x - x * r.y;
    }
    re = sum_of_4(re);
    im = sum_of_4(im);
    if (part == 0)
        U[i] = make_double2(re, im);
}
template <typename T>
__global__ void __launch_bounds__(128) k_fir_taps_outer(T* grad_h, const double2* __restrict__ U,
                                                       const double2* __restrict__ w, int taps, int F, int Q)
{
    stream_order();
    const int t = blockIdx.x * blockDim.x + threadIdx.x, part = t & 3;
    const int P = F / Q, m = min(t >> 2, taps - 1);
    double re = 0;
#pragma unroll 4
    for (int k0 = part; k0 < Q; k0 += 4)
    {
        const double2 u = __ldg(U + k0 * P + (m & (P - 1))), r = __ldg(w + (m * k0 & (F - 1)));
        re += u.x * r.x + u.y * r.y;
    }
    re = sum_of_4(re);
    if (part == 0)
        grad_h[m] = T(re / F);
}

// ---------------------------------------------------------------------------------------------------
// Single precision, where a block would be 8192 samples or more and the overlap is at most half of 4096 (conv_paired): two
// output blocks of a channel as the real and the imaginary part of one 4096-point transform (conv16.cuh).  The taps are
// real, so the product with their spectrum filters both, with no split or merge, and it happens in registers between the
// last forward and the first inverse pass.  Bound by instruction issue, the twiddles' loads (all from the table; with 80
// registers for three CTAs per SM they spill, 283 us) and the latency of the first loads.  64 channels of 2^20 samples,
// 1023 taps: 370 us with one block of 8192 samples through a compile-time 4096-point transform, 250 us so; with powers of
// two table values 226 us, but 1.2 times the relative RMS error of the former (from the table 0.95 times).
// ---------------------------------------------------------------------------------------------------
__device__ __forceinline__ float conv_sample(const float* in, const float* hist, long long i, long long n, long long nhist)
{
    if (i >= 0)
        return i < n ? in[i] : 0.0f;
    return i + nhist >= 0 ? hist[i + nhist] : 0.0f; // the latest sample before the call at hist[nhist - 1]
}

__global__ void __launch_bounds__(fft16::threads, 2) k_conv16(const __grid_constant__ conv_args a)
{
    stream_order();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const fft16 f(smem_raw, a.tw);
    const float* in   = reinterpret_cast<const float*>(a.in) + (long long)blockIdx.y * a.n;
    const float* hist = reinterpret_cast<const float*>(a.hist) + (long long)blockIdx.y * a.nhist;
    float* out        = reinterpret_cast<float*>(a.out) + (long long)blockIdx.y * a.n;
    const int m1 = int(a.m1), bo = int(a.bo);
    const long long first = 2LL * blockIdx.x * bo; // first output of the first block
    const long long start = first - m1;
    cpx<float> v[16];
    if (start >= 0 && start + bo + fft16::N <= a.n)
    {
        const float* x = in + start + f.t;
#pragma unroll
        for (int r = 0; r < 16; r++)
            v[r] = mk<float>(x[256 * r], x[bo + 256 * r]);
    }
    else
    {
#pragma unroll
        for (int r = 0; r < 16; r++)
        {
            const long long i = start + f.t + 256 * r;
            v[r] = mk<float>(conv_sample(in, hist, i, a.n, a.nhist), conv_sample(in, hist, i + bo, a.n, a.nhist));
        }
    }
    f.forward_a(v);
    __syncthreads();
    f.forward_b();
    __syncthreads();
    f.forward_c(v);
    const cpx<float>* H = reinterpret_cast<const cpx<float>*>(a.hspec) + f.t;
#pragma unroll
    for (int u = 0; u < 16; u++)
        v[u] = conj(v[u] * ldg(H + 256 * u));
    f.inverse_c(v);
    __syncthreads();
    f.inverse_b();
    __syncthreads();
    f.inverse_a(v);
    // outputs p >= m1 of the block are samples first + p - m1; the others wrapped around
    const long long left = a.n - first;
#pragma unroll
    for (int r = 0; r < 16; r++)
    {
        const int p = f.t + 256 * r - m1;
        if (p < 0)
            continue;
        if (p < left)
            out[first + p] = v[r].x;
        if (p + bo < left)
            out[first + bo + p] = -v[r].y;
    }
}

// Gradients (see k_fir_bwd) of two blocks of a channel at a time.  With z_g = g_A + i g_B and z_x = x_A + i x_B the sum
// of Z_g conj(Z_x) over all pairs transforms back to the taps gradient in its real part.  x goes first and its 16 bins
// per thread wait in registers while g takes the buffer; the next pair's samples of x are loaded during the inverse.
__global__ void __launch_bounds__(fft16::threads, 2) k_fir16_bwd(const __grid_constant__ fir_bwd_args a)
{
    stream_order();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const fft16 f(smem_raw, a.tw);
    cpx<float>* acc     = reinterpret_cast<cpx<float>*>(smem_raw) + fft16::elems + f.t; // bin u at 256 u
    const cpx<float>* H = reinterpret_cast<const cpx<float>*>(a.hspec) + f.t;
    const bool want_x = a.grad_x != nullptr, want_h = a.partial != nullptr;
    const int bo = int(a.bo);
    const long long pairs = (a.blocks + 1) / 2, total = pairs * a.channels;
    if (want_h)
#pragma unroll
        for (int u = 0; u < 16; u++)
            acc[256 * u] = mk<float>(0, 0);
    const auto load = [&](cpx<float>(&v)[16], const void* base, long long b, int count)
    {
        // samples [t0, t0 + count) and [t0 + bo, t0 + bo + count) of the pair b's channel, zero beyond them
        const long long ch = b / pairs, t0 = 2 * (b - ch * pairs) * bo;
        const float* x  = reinterpret_cast<const float*>(base) + ch * a.n + t0 + f.t;
        const long long left = a.n - t0 - f.t;
#pragma unroll
        for (int r = 0; r < 16; r++)
        {
            const int i   = 256 * r;
            const bool in = i + f.t < count;
            v[r]          = mk<float>(in && i < left ? x[i] : 0.0f, in && i + bo < left ? x[i + bo] : 0.0f);
        }
    };
    cpx<float> px[16];
    if (want_h && blockIdx.x < total)
        load(px, a.x, blockIdx.x, bo);
    for (long long b = blockIdx.x; b < total; b += gridDim.x)
    {
        cpx<float> v[16];
        load(v, a.grad_y, b, fft16::N);
        if (want_h)
        {
            f.forward_a(px);
            __syncthreads();
            f.forward_b();
            __syncthreads();
            f.forward_c(px);
            __syncthreads();
        }
        f.forward_a(v);
        __syncthreads();
        f.forward_b();
        __syncthreads();
        f.forward_c(v);
        if (want_h)
#pragma unroll
            for (int u = 0; u < 16; u++)
                acc[256 * u] = acc[256 * u] + v[u] * conj(px[u]);
        if (want_h && b + gridDim.x < total)
            load(px, a.x, b + gridDim.x, bo);
        if (want_x)
        {
#pragma unroll
            for (int u = 0; u < 16; u++)
                v[u] = conj(v[u] * conj(ldg(H + 256 * u)));
            f.inverse_c(v);
            __syncthreads();
            f.inverse_b();
            __syncthreads();
            f.inverse_a(v);
            const long long ch = b / pairs, t0 = 2 * (b - ch * pairs) * bo, left = a.n - t0;
            float* gx = reinterpret_cast<float*>(a.grad_x) + ch * a.n + t0;
#pragma unroll
            for (int r = 0; r < 16; r++)
            {
                const int p = f.t + 256 * r;
                if (p >= bo)
                    continue;
                if (p < left)
                    gx[p] = v[r].x;
                if (p + bo < left)
                    gx[p + bo] = -v[r].y;
            }
        }
        __syncthreads();
    }
    if (want_h)
    {
        cpx<float>* p = reinterpret_cast<cpx<float>*>(a.partial) + (long long)blockIdx.x * fft16::N + f.t;
#pragma unroll
        for (int u = 0; u < 16; u++)
            p[256 * u] = acc[256 * u];
    }
}

// new_hist[i] = i + n < m1 ? old_hist[i + n] : in[i + n - m1]
template <typename T>
__global__ void k_hist_update(const T* hold, T* hnew, const T* in, long long n,
                              long long m1, int channels)
{
    stream_order();
    const long long total = m1 * channels;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x)
    {
        const long long ch = i / m1, e = i - ch * m1;
        const long long s  = e + n;
        hnew[i]            = s < m1 ? hold[ch * m1 + s] : in[ch * n + (s - m1)];
    }
}

template <typename K, typename... Args>
static cudaError_t conv_go(K kernel, dim3 grid, int threads, size_t smem, cudaStream_t st, Args... args)
{
    if (smem > 48 * 1024)
    {
        const cudaError_t e = prepare_launch(reinterpret_cast<const void*>(kernel), threads, int(smem));
        if (e != cudaSuccess)
            return e;
    }
    return launch_kernel(kernel, grid, threads, smem, st, args...);
}

template <typename T>
cudaError_t launch_conv_os(const conv_args& a, long long nblocks, cudaStream_t st)
{
    if constexpr (std::is_same<T, float>::value)
        if (a.fft.paired)
            return conv_go(k_conv16, dim3(unsigned((nblocks + 1) / 2), unsigned(a.channels)), fft16::threads,
                           fft16::elems * sizeof(cpx<float>), st, a);
    return conv_dispatch<T>(a.fft,
                            [&](auto p)
                            {
                                return conv_go(k_conv_os<typename decltype(p)::type>,
                                               dim3(unsigned(nblocks), unsigned(a.channels)), a.fft.threads,
                                               size_t(a.fft.elems) * 2 * sizeof(T), st, a);
                            });
}

template <typename T>
cudaError_t launch_hist_update(const void* hold, void* hnew, const void* in, long long n, long long m1, int channels,
                               cudaStream_t st)
{
    const long long total = m1 * channels;
    if (total <= 0)
        return cudaSuccess;
    const long long blocks = std::min<long long>((total + 255) / 256, 4096);
    return launch_kernel(k_hist_update<T>, dim3(unsigned(blocks)), 256, 0, st, static_cast<const T*>(hold),
                         static_cast<T*>(hnew), static_cast<const T*>(in), n, m1, channels);
}

// ------------------------------------------------------------------------------------------------------
// conv_filter
// ------------------------------------------------------------------------------------------------------

static size_t next_pow2(size_t x)
{
    size_t p = 1;
    while (p < x)
        p <<= 1;
    return p;
}

// Largest one-CTA real FFT of the convolution kernels.
template <typename T>
static size_t conv_fft_max()
{
    return sizeof(T) == 4 ? 32768 : 16384;
}

template <typename T>
fir_tables<T>::fir_tables(size_t f, bool paired)
{
    if (paired)
    {
        fft.paired   = true;
        const auto t = pass_twiddles<T>({ 16, 16, 16 });
        tw.upload(t.data(), t.size() * sizeof(t[0]));
        return;
    }
    const int c = int(f / 2);
    std::vector<int> rad;
#define KFR_GPU_CONV_CT_OF(N, TS, ...)                                                                     \
    if (sizeof(T) == 4 && c == N)                                                                          \
    {                                                                                                      \
        rad         = { __VA_ARGS__ };                                                                     \
        fft.ct      = N;                                                                                   \
        fft.threads = TS;                                                                                  \
        fft.elems   = (ct_group_stride_f32(N, TS) + 1) / 2 * 2;                                            \
    }
    KFR_CT_CONV_F32(KFR_GPU_CONV_CT_OF)
#undef KFR_GPU_CONV_CT_OF
    if (!fft.ct)
    {
        rad         = rp_radices(c);
        fft.rp      = rp_build(rad, RP_SIGNALS, 1, int(2 * sizeof(T)), true);
        fft.elems   = (fft.rp.elems + 1) / 2 * 2;
        fft.threads = (std::max(rp_threads_needed(fft.rp, 1, true), std::min(c, 64)) + 31) / 32 * 32;
    }
    const auto t = pass_twiddles<T>(rad);
    tw.upload(t.data(), t.size() * sizeof(t[0]));
    std::vector<std::complex<T>> rt(c + 1);
    for (int k = 0; k <= c; k++)
    {
        const auto w = twiddle(k, (long long)f);
        rt[k]        = std::complex<T>(T(w.real()), T(w.imag()));
    }
    rtw.upload(rt.data(), rt.size() * sizeof(rt[0]));
}

template <typename T>
void fir_tables<T>::roots64(size_t f)
{
    std::vector<std::complex<double>> w(f);
    for (size_t j = 0; j < f; j++)
        w[j] = twiddle((long long)j, (long long)f);
    w64.upload(w.data(), w.size() * sizeof(w[0]));
}

template struct fir_tables<float>;
template struct fir_tables<double>;

// Samples of a block for an overlap of m1 samples: at least 8 times it (at most 1/8 of each block re-reads the overlap;
// measured 0.390 -> 0.374 ms against 4x for 64 channels of 2^20 samples and 1023 taps) and twice the caller's block.
template <typename T>
static size_t conv_block_size(size_t m1, size_t block)
{
    return std::min(std::max({ next_pow2(8 * m1), 2 * next_pow2(block ? block : 1024), size_t(64) }), conv_fft_max<T>());
}

// Whether blocks run in pairs through 4096-point transforms.  Up to half of a pair's block re-reads the overlap, where the
// self-sorting transforms of 16384 samples begin to need fewer instructions.  Below blocks of 8192 samples a pair would be
// longer than the block it replaces: its rounding errors are larger (F = 2048: 1.7e-7 -> 2.3e-7 relative RMS) and a sample
// that is infinite or very loud reaches more outputs (2 (4096 - m1) instead of F - m1).
template <typename T>
static bool conv_paired(size_t m1, size_t block)
{
    return sizeof(T) == 4 && m1 <= fft16::N / 2 && conv_block_size<T>(m1, block) >= 2 * fft16::N;
}

// FFT length for an overlap of m1 samples.
template <typename T>
static size_t conv_fft_size(size_t m1, size_t block)
{
    return conv_paired<T>(m1, block) ? size_t(fft16::N) : conv_block_size<T>(m1, block);
}

template <typename T>
conv_filter<T>::conv_filter(const T* taps, size_t ntaps, size_t block_size, int channels)
    : m_(ntaps), channels_(channels)
{
    if (channels < 1)
        throw std::invalid_argument("convolution filter needs at least one channel");
    std::vector<T> h(ntaps);
    if (ntaps)
    {
        if (!taps)
            throw std::invalid_argument("taps pointer is NULL");
        cudaPointerAttributes pa;
        const bool dev = cudaPointerGetAttributes(&pa, taps) == cudaSuccess &&
                         (pa.type == cudaMemoryTypeDevice || pa.type == cudaMemoryTypeManaged);
        cudaGetLastError();
        check(cudaMemcpy(h.data(), taps, ntaps * sizeof(T), dev ? cudaMemcpyDeviceToHost : cudaMemcpyHostToHost),
              "copy taps");
    }
    const size_t m1 = ntaps ? ntaps - 1 : 0;
    const size_t f = conv_fft_size<T>(m1, block_size);
    const size_t hb = std::max<size_t>(1, m1 * size_t(channels)) * sizeof(T);
    hist_[0].alloc(hb);
    hist_[1].alloc(hb);
    if (m1 >= f / 2 && !conv_paired<T>(m1, block_size))
    {
        // long mode: the taps stay on the device for whole-call convolutions
        long_ = true;
        f_ = c_ = bo_ = 0;
        htaps_.upload(h.data(), ntaps * sizeof(T));
        reset();
        return;
    }
    f_  = f;
    c_  = f / 2;
    const bool paired = conv_paired<T>(m1, block_size);
    bo_ = paired ? f - m1 : f - (m1 + 1) / 2 * 2; // unpaired blocks start at even samples
    tables_.reset(new fir_tables<T>(f, paired));
    // taps spectrum FFT_F(h padded) / F, bins 0..c (set_data, src/dft/convolution-impl.cpp:53-71)
    std::vector<std::complex<double>> a(f, { 0.0, 0.0 });
    for (size_t i = 0; i < ntaps; i++)
        a[i] = double(h[i]);
    host_fft_pow2(a);
    // (paired blocks: every bin, in fft16_place order)
    std::vector<std::complex<T>> hs(paired ? f : c_ + 1);
    for (size_t k = 0; k < hs.size(); k++)
        hs[paired ? fft16_place(int(k)) : int(k)] = std::complex<T>(T(a[k].real() / double(f)), T(a[k].imag() / double(f)));
    hspec_.upload(hs.data(), hs.size() * sizeof(std::complex<T>));
    reset();
}

template <typename T>
void conv_filter<T>::reset()
{
    check(cudaMemset(hist_[0].get(), 0, hist_[0].size()), "reset filter state");
    check(cudaMemset(hist_[1].get(), 0, hist_[1].size()), "reset filter state");
    cur_ = 0;
}

template <typename T>
int conv_filter<T>::launches(size_t n) const
{
    if (long_ && n)
        return 2 + 8 * channels_; // per channel: two pads, two forward and one inverse real FFT, the product
    return (n && m_) ? (m_ > 1 ? 2 : 1) : (n ? 1 : 0);
}

template <typename T>
void conv_filter<T>::process(T* out, const T* in, size_t n, cudaStream_t st)
{
    if (n == 0)
        return;
    if (m_ == 0)
    {
        check(cudaMemsetAsync(out, 0, n * channels_ * sizeof(T), st), "zero output");
        return;
    }
    const long long m1 = (long long)m_ - 1;
    if (long_)
    {
        // y = ([history, input] * taps)[m1 + t], t < n, one real-FFT convolution per channel
        const long long ulen = m1 + (long long)n;
        lin_.ensure(size_t(ulen) * sizeof(T));
        lout_.ensure(size_t(ulen + (long long)m_ - 1) * sizeof(T));
        T* u = static_cast<T*>(lin_.get());
        T* y = static_cast<T*>(lout_.get());
        for (int ch = 0; ch < channels_; ch++)
        {
            check(cudaMemcpyAsync(u, static_cast<const T*>(hist_[cur_].get()) + ch * m1, size_t(m1) * sizeof(T),
                                  cudaMemcpyDeviceToDevice, st),
                  "copy filter history");
            check(cudaMemcpyAsync(u + m1, in + ch * (long long)n, n * sizeof(T), cudaMemcpyDeviceToDevice, st),
                  "copy filter input");
            convolve_device<T>(y, u, ulen, htaps_.get(), (long long)m_, false, 0, st);
            check(cudaMemcpyAsync(out + ch * (long long)n, y + m1, n * sizeof(T), cudaMemcpyDeviceToDevice, st),
                  "copy filter output");
        }
        check(launch_hist_update<T>(hist_[cur_].get(), hist_[1 - cur_].get(), in, (long long)n, m1, channels_, st),
              "launch history update");
        cur_ = 1 - cur_;
        return;
    }
    conv_args a;
    a.in       = in;
    a.out      = out;
    a.hist     = hist_[cur_].get();
    a.n        = (long long)n;
    a.nhist    = m1;
    a.m1       = tables_->fft.paired ? m1 : (m1 + 1) / 2 * 2;
    a.bo       = (long long)bo_;
    a.channels = channels_;
    a.hspec    = hspec_.get();
    a.rtw      = tables_->rtw.get();
    a.tw       = tables_->tw.get();
    a.fft      = tables_->fft;
    const long long nbl = ((long long)n + (long long)bo_ - 1) / (long long)bo_;
    check(launch_conv_os<T>(a, nbl, st), "launch convolution");
    if (m1 > 0)
    {
        check(launch_hist_update<T>(hist_[cur_].get(), hist_[1 - cur_].get(), in, (long long)n, m1, channels_, st),
              "launch history update");
        cur_ = 1 - cur_;
    }
}

// ------------------------------------------------------------------------------------------------------
// gradients
// ------------------------------------------------------------------------------------------------------

template <typename T>
bool fir_backward_blocks(const T* taps, long long ntaps, long long channels, long long n, const T* x, const T* grad_y,
                         T* grad_x, T* grad_h, cudaStream_t st)
{
    const size_t m1 = size_t(ntaps - 1);
    const bool paired = conv_paired<T>(m1, 1024);
    // the gradient kernel holds two spectra and a sum: half the one-CTA length
    const size_t f = std::min(conv_fft_size<T>(m1, 1024), conv_fft_max<T>() / 2);
    if (m1 >= f / 2 && !paired)
        return false;
    const auto tab = plan_cache::instance().fir<T>((long long)f, paired);
    const int c    = int(f / 2);
    const int bins = paired ? int(f) : c + 1; // bins of a spectrum
    fir_bwd_args a;
    a.x        = x;
    a.grad_y   = grad_y;
    a.grad_x   = grad_x;
    a.n        = n;
    a.bo       = (long long)(f - (paired ? m1 : (m1 + 1) / 2 * 2));
    a.blocks   = (n + a.bo - 1) / a.bo;
    a.channels = channels;
    a.rtw      = tab->rtw.get();
    a.tw       = tab->tw.get();
    a.fft      = tab->fft;
    a.elems    = tab->fft.elems;
    const int threads     = paired ? fft16::threads : a.fft.threads;
    const size_t smem     = paired ? (size_t(fft16::elems) + fft16::N) * 2 * sizeof(T) : (2 * size_t(a.elems) + c + 1) * 2 * sizeof(T);
    const long long total = (paired ? (a.blocks + 1) / 2 : a.blocks) * channels;
    // the taps' inner sums of about the square root of F rows
    int Q = 1;
    while (Q * Q < int(f))
        Q <<= 1;
    const auto bwd = conv_dispatch<T>(a.fft, [](auto p) { return &k_fir_bwd<typename decltype(p)::type>; });
    const void* kernel = reinterpret_cast<const void*>(bwd);
    if constexpr (std::is_same<T, float>::value)
        if (paired)
            kernel = reinterpret_cast<const void*>(k_fir16_bwd);
    int per_sm = 0;
    check(prepare_launch(kernel, threads, int(smem), &per_sm), "prepare FIR backward");
    const int grid = int(std::min<long long>(total, (long long)per_sm * device_sm_count()));
    const size_t cpx_b  = 2 * sizeof(T);
    const size_t hs_b   = (size_t(bins) * cpx_b + 255) / 256 * 256;
    const size_t in_b   = f * sizeof(double2);
    const size_t part_b = grad_h ? size_t(grid) * bins * cpx_b : 0;
    // the blocks read gradients that other blocks overwrite when grad_x shares memory with an input
    const auto overlaps = [&](const void* p)
    {
        const char *u = reinterpret_cast<const char*>(grad_x), *v = static_cast<const char*>(p);
        const size_t bytes = size_t(channels * n) * sizeof(T);
        return u && v && u < v + bytes && v < u + bytes;
    };
    const bool staged = overlaps(grad_y) || (grad_h && overlaps(x));
    workspace ws(2 * hs_b + in_b + part_b + (staged ? size_t(channels * n) * sizeof(T) : 0), st);
    char* H      = static_cast<char*>(ws.get());
    char* sum    = H + hs_b;
    char* inner  = sum + hs_b;
    char* parts  = inner + in_b;
    a.hspec      = H;
    a.partial    = grad_h ? parts : nullptr;
    if (staged)
        a.grad_x = parts + part_b;
    if (grad_x)
    {
        const double2* w = static_cast<const double2*>(tab->w64.get());
        launch_kernel(k_fir_spec_inner<T>, dim3(unsigned((f + 127) / 128)), 128, 0, st,
                      reinterpret_cast<double2*>(inner), taps, w, int(ntaps), int(f), Q);
        launch_kernel(k_fir_spec_outer<T>, dim3(unsigned((4 * (c + 1) + 127) / 128)), 128, 0, st, reinterpret_cast<cpx<T>*>(H),
                      reinterpret_cast<const double2*>(inner), w, int(ntaps), int(f), Q, paired);
        check(cudaGetLastError(), "taps spectrum");
    }
    if (paired)
    {
        if constexpr (std::is_same<T, float>::value)
            check(conv_go(k_fir16_bwd, dim3(unsigned(grid)), threads, smem, st, a), "launch FIR backward");
    }
    else
        check(conv_go(bwd, dim3(unsigned(grid)), threads, smem, st, a), "launch FIR backward");
    if (grad_h)
    {
        const double2* w = static_cast<const double2*>(tab->w64.get());
        launch_kernel(k_fir_reduce<T>, dim3(unsigned((bins + 31) / 32)), 256, 0, st, reinterpret_cast<cpx<T>*>(sum),
                      reinterpret_cast<const cpx<T>*>(parts), grid, bins);
        launch_kernel(k_fir_taps_inner<T>, dim3(unsigned((4 * f + 127) / 128)), 128, 0, st, reinterpret_cast<double2*>(inner),
                      reinterpret_cast<const cpx<T>*>(sum), w, int(f), Q, paired);
        launch_kernel(k_fir_taps_outer<T>, dim3(unsigned((4 * ntaps + 127) / 128)), 128, 0, st, grad_h,
                      reinterpret_cast<const double2*>(inner), w, int(ntaps), int(f), Q);
        check(cudaGetLastError(), "launch FIR backward (taps)");
    }
    if (staged)
        check(cudaMemcpyAsync(grad_x, a.grad_x, size_t(channels * n) * sizeof(T), cudaMemcpyDeviceToDevice, st),
              "copy signal gradient");
    return true;
}

template bool fir_backward_blocks<float>(const float*, long long, long long, long long, const float*, const float*,
                                         float*, float*, cudaStream_t);
template bool fir_backward_blocks<double>(const double*, long long, long long, long long, const double*, const double*,
                                          double*, double*, cudaStream_t);
template class conv_filter<float>;
template class conv_filter<double>;
template cudaError_t launch_conv_os<float>(const conv_args&, long long, cudaStream_t);
template cudaError_t launch_conv_os<double>(const conv_args&, long long, cudaStream_t);

} // namespace kfr_gpu
