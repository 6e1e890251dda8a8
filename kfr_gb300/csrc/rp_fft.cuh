// Runtime-length block FFT over a tile of signals in one shared buffer (plans and layouts: rp.hpp).
//
// What bounds it: instruction issue.  A pass spends, per element, one shared load, one shared store, two
// address steps, the codelet and a twiddle product whose power comes from one table value per butterfly
// (binary powering), close to the compile-time passes: the butterfly's two addresses are computed once and
// the rest are constant steps, with no padding arithmetic per element (rp.hpp), no per-signal thread groups
// (the tile's butterflies are dealt to the threads in one sequence, so any radix keeps all threads busy) and
// no register array carried across the radix switch.  The first pass reads its inputs through a functor
// (global memory, with any pre-processing) and the last pass writes through one, so a transform of two passes
// crosses shared memory once.  Middle passes are in place: each thread holds rp_held(R) butterflies across
// one barrier, which halves the shared memory of ping-pong buffers and so doubles the CTAs whose global
// accesses overlap.  Figures: k_rp_c2c, k_rp_cols (rp_kernels.cuh).
#pragma once

#include "fft_device.cuh"
#include "rp.hpp"

namespace kfr_gpu
{

struct rp_lane
{
    int g, j, q, k; // signal of the tile, butterfly, j = q ns + k
};

// CT: the pass and shift are compile-time constants (plain divisions fold).
template <bool CT = false>
__device__ __forceinline__ rp_lane rp_map(const rp_pass& p, const int shift, const int J)
{
    rp_lane l;
    if constexpr (CT)
    {
        l.g = p.fast ? J & ((1 << shift) - 1) : int(uint32_t(J) / uint32_t(p.nbf));
        l.j = p.fast ? J >> shift : int(uint32_t(J) % uint32_t(p.nbf));
        l.q = int(uint32_t(l.j) / uint32_t(p.ns));
        l.k = int(uint32_t(l.j) % uint32_t(p.ns));
        return l;
    }
    if (p.fast)
    {
        l.g = J & ((1 << shift) - 1);
        l.j = J >> shift;
    }
    else
    {
        l.g = p.mg ? int(__umulhi(uint32_t(J), p.mg)) : J;
        l.j = J - l.g * p.nbf;
    }
    l.q = p.mq ? int(__umulhi(uint32_t(l.j), p.mq)) : l.j;
    l.k = l.j - l.q * p.ns;
    return l;
}

// TABLE: every power from the table (double precision always: FP64 products are slow on this part).  Powers of one or
// two table values round again with each product.
template <typename T, int R, bool TABLE>
__device__ __forceinline__ void rp_twiddle(cpx<T> (&v)[R], const rp_pass& p, const cpx<T>* __restrict__ tw, const int k)
{
    if constexpr (R == 1)
        return;
    if (p.ns == 1)
        return;
    const cpx<T>* t = tw + p.tw_off + k;
    if constexpr (sizeof(T) == 4 && !TABLE)
    {
        if constexpr (R > 4)
            twiddle_powers4<T, R>(v, ldg(t), ldg(t + 3 * p.ns));
        else
            twiddle_powers<T, R>(v, ldg(t));
    }
    else
    {
#pragma unroll
        for (int r = 1; r < R; r++)
            v[r] = v[r] * ldg(t + (r - 1) * p.ns);
    }
}

// Shared-memory ends of a pass.
template <typename T>
struct rp_smem
{
    cpx<T>* buf;
    __device__ __forceinline__ cpx<T>* src(const rp_pass& p, const rp_lane& l) const
    {
        return buf + l.j * p.ld_e + l.q * p.ld_q + l.g * p.ld_g;
    }
    __device__ __forceinline__ cpx<T>* dst(const rp_pass& p, const rp_lane& l) const
    {
        return buf + l.k * p.st_e + l.q * p.st_q + l.g * p.st_g;
    }
};

// First pass: inputs ld(g, i), outputs to shared memory; prep(g, j, step, v) sees a butterfly's inputs v[r]
// (input j + r step) once all of them are loaded.
template <typename T, int R, bool CT = false, class LD, class PREP>
__device__ __forceinline__ void rp_first(const rp_pass& p, const int shift, const int total, const rp_smem<T> sm,
                                         const LD& ld, const PREP& prep)
{
    for (int J = threadIdx.x; J < total; J += blockDim.x)
    {
        const rp_lane l = rp_map<CT>(p, shift, J);
        cpx<T> v[R];
#pragma unroll
        for (int r = 0; r < R; r++)
            v[r] = ld(l.g, l.j + r * p.nbf);
        prep(l.g, l.j, p.nbf, v);
        dft_codelet<T, R>(v);
        cpx<T>* d = sm.dst(p, l);
#pragma unroll
        for (int r = 0; r < R; r++)
            d[r * p.st_r] = v[codelet_out<R>(r)];
    }
}

// Last pass: inputs from shared memory; fin(g, k, step, o) sees the butterfly's outputs o[r] (output k + r step)
// before st(g, i, x) stores them.
template <typename T, int R, bool CT = false, bool TABLE = false, class ST, class FIN>
__device__ __forceinline__ void rp_last(const rp_pass& p, const int shift, const int total, const rp_smem<T> sm,
                                        const cpx<T>* __restrict__ tw, const ST& st, const FIN& fin)
{
    for (int J = threadIdx.x; J < total; J += blockDim.x)
    {
        const rp_lane l   = rp_map<CT>(p, shift, J);
        const cpx<T>* s = sm.src(p, l);
        cpx<T> v[R];
#pragma unroll
        for (int r = 0; r < R; r++)
            v[r] = s[r * p.ld_r];
        rp_twiddle<T, R, TABLE>(v, p, tw, l.k);
        dft_codelet<T, R>(v);
        cpx<T> o[R];
#pragma unroll
        for (int r = 0; r < R; r++)
            o[r] = v[codelet_out<R>(r)];
        fin(l.g, l.k, p.ns, o);
#pragma unroll
        for (int r = 0; r < R; r++)
            st(l.g, l.k + r * p.ns, o[r]);
    }
}

// In-place pass: the thread's butterflies are held in registers across a barrier (rp_threads_needed).
template <typename T, int R, int H, bool CT = false, bool TABLE = false>
__device__ __forceinline__ void rp_mid(const rp_pass& p, const int shift, const int total, const rp_smem<T> sm,
                                       const cpx<T>* __restrict__ tw)
{
    constexpr int NB = rp_held(R, H);
    cpx<T> v[NB][R];
#pragma unroll
    for (int b = 0; b < NB; b++)
    {
        const int J = threadIdx.x + b * blockDim.x;
        if (J < total)
        {
            const rp_lane l   = rp_map<CT>(p, shift, J);
            const cpx<T>* s = sm.src(p, l);
#pragma unroll
            for (int r = 0; r < R; r++)
                v[b][r] = s[r * p.ld_r];
            rp_twiddle<T, R, TABLE>(v[b], p, tw, l.k);
            dft_codelet<T, R>(v[b]);
        }
        else
        {
            // defined on every path: otherwise ptxas takes the values of all radix cases as live around the
            // pass loop and spills them (1500 bytes; 3600 points 20% slower)
#pragma unroll
            for (int r = 0; r < R; r++)
                v[b][r] = mk<T>(0, 0);
        }
    }
    __syncthreads();
#pragma unroll
    for (int b = 0; b < NB; b++)
    {
        const int J = threadIdx.x + b * blockDim.x;
        if (J < total)
        {
            const rp_lane l = rp_map<CT>(p, shift, J);
            cpx<T>* d     = sm.dst(p, l);
#pragma unroll
            for (int r = 0; r < R; r++)
                d[r * p.st_r] = v[b][codelet_out<R>(r)];
        }
    }
}

// In-place pass of a prime radix above 13: the inputs are twiddled where they lie, then each thread holds up to
// H outputs o = s nbf total + J, each a dot product of a butterfly's inputs with the roots W_R^{s r}.
template <typename T, int H>
__device__ __forceinline__ void rp_prime(const rp_pass& p, const int shift, const int total, const rp_smem<T> sm,
                                         const cpx<T>* __restrict__ tw)
{
    const int R = p.radix;
    if (p.ns > 1)
    {
        // input r >= 1 of each butterfly by itself: a tile has few butterflies of a large radix
        for (int o = threadIdx.x; o < (R - 1) * total; o += blockDim.x)
        {
            const int r     = o / total; // r + 1 of the butterfly
            const rp_lane l = rp_map(p, shift, o - r * total);
            cpx<T>* s       = sm.src(p, l) + (r + 1) * p.ld_r;
            *s              = *s * ldg(tw + p.tw_off + r * p.ns + l.k);
        }
        __syncthreads();
    }
    constexpr int E  = H;
    const cpx<T>* wr = tw + p.wr_off;
    cpx<T> v[E];
#pragma unroll
    for (int e = 0; e < E; e++)
    {
        const int o = threadIdx.x + e * blockDim.x;
        const int q = o / total;
        if (q < R)
        {
            const cpx<T>* s = sm.src(p, rp_map(p, shift, o - q * total));
            cpx<T> acc      = s[0];
            int m           = 0;
#pragma unroll 1
            for (int r = 1; r < R; r++)
            {
                m += q;
                if (m >= R)
                    m -= R;
                acc = acc + s[r * p.ld_r] * ldg(wr + m);
            }
            v[e] = acc;
        }
        else
            v[e] = mk<T>(0, 0);
    }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < E; e++)
    {
        const int o = threadIdx.x + e * blockDim.x;
        const int q = o / total;
        if (q < R)
            sm.dst(p, rp_map(p, shift, o - q * total))[q * p.st_r] = v[e];
    }
}

// Element i of the array at p whose elements are `bytes` (32 or 64 bits wide) apart: one or two wide
// multiply-adds.
template <typename C, typename N>
__device__ __forceinline__ C* rp_at(C* p, int i, N bytes)
{
    using B = std::conditional_t<std::is_const_v<C>, const char, char>;
    return reinterpret_cast<C*>(reinterpret_cast<B*>(p) + (unsigned long long)(uint32_t(i)) * bytes);
}

#define KFR_GPU_RP_CODELETS(X) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13) X(14) X(15) X(16)
#define KFR_GPU_RP_RADICES(X) X(1) KFR_GPU_RP_CODELETS(X) // the ends of a transform: radix 1 copies

struct rp_no_hook
{
    template <class O>
    __device__ __forceinline__ void operator()(int, int, int, O&) const
    {
    }
};

// The whole transform of `nsig` signals.  D: anything with n, npass, shift and pass[] (a kernel parameter, or a
// copy in shared memory); every thread of the CTA takes part.  ld(g, i) reads input i of signal g, st(g, i, x)
// takes output i; work that depends on uniform flags belongs in the hooks (rp_first, rp_last), which run once
// per butterfly.  Every input is read before the first output is stored when npass > 1 (or, for one pass,
// by the thread that stores the signal's outputs), so the two may be the same memory.  Shared memory is free
// again only after a barrier.
template <typename T, int H = kRpHold, bool TABLE = false, class D, class LD, class ST, class FIN = rp_no_hook, class PREP = rp_no_hook>
__device__ __forceinline__ void rp_run(const D& d, cpx<T>* buf, const int nsig, const cpx<T>* __restrict__ tw,
                                       const LD& ld, const ST& st, const FIN& fin = FIN(),
                                       const PREP& prep = PREP())
{
    const rp_smem<T> sm{ buf };
    const int np = d.npass, sh = d.shift;
    {
        const rp_pass& p = d.pass[0];
        const int total  = nsig * p.nbf;
        switch (p.radix)
        {
#define KFR_GPU_RP_CASE(R)                                                                                 \
    case R: rp_first<T, R>(p, sh, total, sm, ld, prep); break;
            KFR_GPU_RP_RADICES(KFR_GPU_RP_CASE)
#undef KFR_GPU_RP_CASE
        default: break;
        }
    }
    __syncthreads();
#pragma unroll 1
    for (int i = 1; i + 1 < np; i++)
    {
        const rp_pass& p = d.pass[i];
        const int total  = nsig * p.nbf;
        switch (p.radix)
        {
#define KFR_GPU_RP_CASE(R)                                                                                 \
    case R: rp_mid<T, R, H, false, TABLE>(p, sh, total, sm, tw); break;
            KFR_GPU_RP_CODELETS(KFR_GPU_RP_CASE)
#undef KFR_GPU_RP_CASE
        default: rp_prime<T, H>(p, sh, total, sm, tw); break;
        }
        __syncthreads();
    }
    if (np == 1)
    {
        // one codelet: its outputs lie in natural order
        const rp_pass& p = d.pass[0];
        const int n      = p.radix;
        for (int i = threadIdx.x; i < nsig * n; i += blockDim.x)
        {
            const int g = p.fast ? i & ((1 << sh) - 1) : i / n;
            const int k = p.fast ? i >> sh : i - g * n;
            cpx<T> o[1] = { buf[k * p.st_r + g * p.st_g] };
            fin(g, k, 0, o);
            st(g, k, o[0]);
        }
        return;
    }
    const rp_pass& p = d.pass[np - 1];
    const int total  = nsig * p.nbf;
    switch (p.radix)
    {
#define KFR_GPU_RP_CASE(R)                                                                                 \
    case R: rp_last<T, R, false, TABLE>(p, sh, total, sm, tw, st, fin); break;
        KFR_GPU_RP_RADICES(KFR_GPU_RP_CASE)
#undef KFR_GPU_RP_CASE
    default: break;
    }
}

// Compile-time descriptor of the radices Rs over a tile of S signals of RP_COLS or RP_ROWS (as rp_build, with `pad`
// spare slots after each group of the first pass and none after the others, whose stores are contiguous).
template <rp_layout L, int S, int PAD, int... Rs>
struct rp_ct
{
    static constexpr int npass = sizeof...(Rs);
    static constexpr rp_desc make()
    {
        constexpr int rad[] = { Rs... };
        rp_desc d{};
        d.npass = npass;
        d.n     = (Rs * ...);
        d.hold  = kRpHold;
        while ((1 << d.shift) < S)
            d.shift++;
        int ns = 1, off = 0;
        for (int i = 0; i < npass; i++)
        {
            rp_pass& p = d.pass[i];
            p.radix    = rad[i];
            p.ns       = ns;
            p.nbf      = d.n / rad[i];
            p.fast     = L == RP_COLS || i > 0;
            p.tw_off   = off;
            if (ns > 1)
                off += ns * (rad[i] - 1);
            ns *= rad[i];
        }
        for (int i = 0; i + 1 < npass; i++)
        {
            rp_pass &a = d.pass[i], &b = d.pass[i + 1];
            const int nn = a.ns * a.radix, pad = i == 0 ? PAD : 0;
            a.st_e  = S;
            a.st_q  = nn * S + pad;
            a.st_g  = 1;
            a.st_r  = a.ns * S;
            b.ld_e  = S;
            b.ld_q  = pad;
            b.ld_g  = 1;
            b.ld_r  = b.nbf * S + b.nbf / nn * pad;
            d.elems = d.elems > d.n / nn * a.st_q ? d.elems : d.n / nn * a.st_q;
        }
        return d;
    }
    static constexpr rp_desc d = make();
    static constexpr int threads()
    {
        int t = 128;
        for (int i = 1; i + 1 < npass; i++)
        {
            const int h = rp_held(d.pass[i].radix, kRpHold), need = (S * d.pass[i].nbf + h - 1) / h;
            t = t > need ? t : need;
        }
        return (t + 31) / 32 * 32;
    }
};

// rp_run with every index a constant.
template <typename T, class C, int I = 1, class LD, class ST, class FIN = rp_no_hook>
__device__ __forceinline__ void rp_run_ct(cpx<T>* buf, const cpx<T>* __restrict__ tw, const LD& ld, const ST& st,
                                          const FIN& fin = FIN())
{
    constexpr rp_desc D = C::d;
    constexpr int S     = 1 << D.shift;
    const rp_smem<T> sm{ buf };
    if constexpr (I == 1)
    {
        constexpr rp_pass p = D.pass[0];
        rp_first<T, p.radix, true>(p, D.shift, S * p.nbf, sm, ld, rp_no_hook{});
        __syncthreads();
    }
    constexpr rp_pass p = D.pass[I];
    if constexpr (I + 1 < D.npass)
    {
        rp_mid<T, p.radix, kRpHold, true>(p, D.shift, S * p.nbf, sm, tw);
        __syncthreads();
        rp_run_ct<T, C, I + 1>(buf, tw, ld, st, fin);
    }
    else
        rp_last<T, p.radix, true>(p, D.shift, S * p.nbf, sm, tw, st, fin);
}

// The transform from ld(g, i) to shared memory (output k of signal g in the natural layout of d's last pass).  Ends
// with a barrier.
template <typename T, int H = kRpHold, class D, class LD>
__device__ __forceinline__ void rp_run_in(const D& d, cpx<T>* buf, const int nsig, const cpx<T>* __restrict__ tw,
                                          const LD& ld)
{
    const rp_smem<T> sm{ buf };
    const rp_no_hook none{};
    {
        const rp_pass& p = d.pass[0];
        const int total  = nsig * p.nbf;
        switch (p.radix)
        {
#define KFR_GPU_RP_CASE(R)                                                                                 \
    case R: rp_first<T, R>(p, d.shift, total, sm, ld, none); break;
            KFR_GPU_RP_RADICES(KFR_GPU_RP_CASE)
#undef KFR_GPU_RP_CASE
        default: break;
        }
    }
    __syncthreads();
#pragma unroll 1
    for (int i = 1; i < d.npass; i++)
    {
        const rp_pass& p = d.pass[i];
        const int total  = nsig * p.nbf;
        switch (p.radix)
        {
#define KFR_GPU_RP_CASE(R)                                                                                 \
    case R: rp_mid<T, R, H>(p, d.shift, total, sm, tw); break;
            KFR_GPU_RP_CODELETS(KFR_GPU_RP_CASE)
#undef KFR_GPU_RP_CASE
        default: rp_prime<T, H>(p, d.shift, total, sm, tw); break;
        }
        __syncthreads();
    }
}

// The transform from and to shared memory (natural order at both ends), every pass in place.  Ends with a
// barrier.
template <typename T, int H = kRpHold, class D>
__device__ __forceinline__ void rp_run_smem(const D& d, cpx<T>* buf, const int nsig, const cpx<T>* __restrict__ tw)
{
    const rp_smem<T> sm{ buf };
#pragma unroll 1
    for (int i = 0; i < d.npass; i++)
    {
        const rp_pass& p = d.pass[i];
        const int total  = nsig * p.nbf;
        switch (p.radix)
        {
#define KFR_GPU_RP_CASE(R)                                                                                 \
    case R: rp_mid<T, R, H>(p, d.shift, total, sm, tw); break;
            KFR_GPU_RP_CODELETS(KFR_GPU_RP_CASE)
#undef KFR_GPU_RP_CASE
        default: rp_prime<T, H>(p, d.shift, total, sm, tw); break;
        }
        __syncthreads();
    }
}

} // namespace kfr_gpu
