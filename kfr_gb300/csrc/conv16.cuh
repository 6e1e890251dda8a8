// 4096-point complex FFT of one 256-thread CTA for pointwise work on spectra (convolution), three radix-16 passes in
// place and no reordering: the forward passes (decimation in frequency) leave the bins where they fall, the inverse
// ones (decimation in time) take them from there, and the last forward and the first inverse pass of a thread work on
// the same 16 values, so a spectrum is multiplied in registers.  Against self-sorting passes a convolution block
// crosses shared memory 8 times instead of 12, with 4 barriers instead of 10.
//
// Sample n = n0 + 16 n1 + 256 n2 of a signal; bin k = r + 16 s + 256 u.  Value e = 16 (16 a + b) + c of the buffer lies
// at e + e / 16 (one spare slot every 16 keeps the last pass's rows apart).  tw: the twiddles of the radices
// {16, 16, 16} (pass_twiddles).
#pragma once

#include "fft_device.cuh"

namespace kfr_gpu
{

struct fft16
{
    static constexpr int N = 4096, threads = 256, elems = N + N / 16;
    cpx<float>* const s;
    const cpx<float>* const tw1; // W_256^(k r)
    const cpx<float>* const tw2; // W_4096^(k r)
    const int t;
    __device__ __forceinline__ fft16(void* smem, const void* tw)
        : s(reinterpret_cast<cpx<float>*>(smem)), tw1(reinterpret_cast<const cpx<float>*>(tw)), tw2(tw1 + 15 * 16),
          t(int(threadIdx.x))
    {
    }
    // v[r] *= W^{k r}, every value from the table: t = tw1 or tw2 + k, rows r - 1 of STRIDE values
    template <int STRIDE>
    static __device__ __forceinline__ void twiddle(cpx<float> (&v)[16], const cpx<float>* t)
    {
#pragma unroll
        for (int r = 1; r < 16; r++)
            v[r] = v[r] * ldg(t + (r - 1) * STRIDE);
    }
    static __device__ __forceinline__ void dft(cpx<float> (&v)[16])
    {
        dft_codelet<float, 16>(v);
        cpx<float> o[16];
#pragma unroll
        for (int r = 0; r < 16; r++)
            o[r] = v[codelet_out<16>(r)];
#pragma unroll
        for (int r = 0; r < 16; r++)
            v[r] = o[r];
    }
    // samples v[n2] = x[t + 256 n2]
    __device__ __forceinline__ void forward_a(cpx<float> (&v)[16]) const
    {
        dft(v);
        twiddle<256>(v, tw2 + t);
        cpx<float>* d = s + t + (t >> 4);
#pragma unroll
        for (int r = 0; r < 16; r++)
            d[r * 272] = v[r];
    }
    __device__ __forceinline__ void forward_b() const
    {
        cpx<float>* d = s + (t >> 4) * 272 + (t & 15);
        cpx<float> v[16];
#pragma unroll
        for (int n1 = 0; n1 < 16; n1++)
            v[n1] = d[n1 * 17];
        dft(v);
        twiddle<16>(v, tw1 + (t & 15));
#pragma unroll
        for (int r = 0; r < 16; r++)
            d[r * 17] = v[r];
    }
    // bins v[u] = X[(t >> 4) + 16 (t & 15) + 256 u]
    __device__ __forceinline__ void forward_c(cpx<float> (&v)[16]) const
    {
#pragma unroll
        for (int i = 0; i < 16; i++)
            v[i] = s[t * 17 + i];
        dft(v);
    }
    // The inverse passes run conj(DFT(conj x)): v[u] = conj(Y) of the bins of forward_c; the results come conjugated.
    __device__ __forceinline__ void inverse_c(cpx<float> (&v)[16]) const
    {
        dft(v);
#pragma unroll
        for (int i = 0; i < 16; i++)
            s[t * 17 + i] = v[i];
    }
    __device__ __forceinline__ void inverse_b() const
    {
        cpx<float>* d = s + (t >> 4) * 272 + (t & 15);
        cpx<float> v[16];
#pragma unroll
        for (int r = 0; r < 16; r++)
            v[r] = d[r * 17];
        twiddle<16>(v, tw1 + (t & 15));
        dft(v);
#pragma unroll
        for (int n1 = 0; n1 < 16; n1++)
            d[n1 * 17] = v[n1];
    }
    // v[n2] = conj(y[t + 256 n2])
    __device__ __forceinline__ void inverse_a(cpx<float> (&v)[16]) const
    {
        const cpx<float>* d = s + t + (t >> 4);
#pragma unroll
        for (int r = 0; r < 16; r++)
            v[r] = d[r * 272];
        twiddle<256>(v, tw2 + t);
        dft(v);
    }
};

// Place of bin k in a spectrum stored for forward_c: thread t's u-th bin at t + 256 u.
__host__ __device__ constexpr int fft16_place(int k) { return (k & 15) * 16 + ((k >> 4) & 15) + (k >> 8) * 256; }

} // namespace kfr_gpu
