// FFT convolution filter: the GPU counterpart of convolve_filter<T> (include/kfr/dft/convolution.hpp:98-148,
// src/dft/convolution-impl.cpp:37-84, 134-228).
//
// The reference streams a uniformly partitioned overlap-add, one block at a time, keeping the FFTs of past
// blocks and the overlap as state.  Its output is the causal FIR convolution of everything passed since
// the last reset(): y[n] = sum_{k<M} h[k] x[n-k].  Here every output block of a process() call is computed
// at once by a batched overlap-save: CTA b takes input samples [b*B - (M-1), b*B + B) (the part before the
// call comes from a device history of the last M-1 samples), runs a real FFT of F = B + M - 1 samples (a power of
// two, at least 8 (M - 1) and twice the caller's block size), multiplies by the taps' spectrum (scaled by 1/F, as
// set_data does), runs the inverse, and writes its B valid samples.  Single-precision blocks of 8192 samples and more
// with an overlap of at most 2048 run as pairs of F = 4096 samples through one complex transform instead (conv16.cuh):
// a sample that is infinite or very loud reaches the outputs of both, 2 (4096 - (M - 1)) at most.  State is the M-1
// sample history per channel, so results do not depend on how the input is split into calls.
#pragma once

#include "plan.hpp"

namespace kfr_gpu
{

// The transform of a convolution block: c complex points for F = 2c samples, or pairs of blocks of F = 4096 samples
// through one complex transform (conv16.cuh; spectra then hold all F bins in fft16_place order).
struct conv_fft
{
    bool paired = false;
    int ct      = 0; // unpaired: c of a compile-time transform (KFR_CT_CONV_F32), 0 = rp
    int threads = 0;
    int elems   = 0; // shared complex elements (even)
    rp_desc rp{};
};

// Tables of real FFTs of f samples in the convolution kernels.
template <typename T>
struct fir_tables
{
    fir_tables(size_t f, bool paired);
    void roots64(size_t f); // w64
    conv_fft fft;
    dbuf tw, rtw; // pass twiddles; W_f^k, k <= f / 2 (unpaired)
    dbuf w64;     // W_f^j, j < f, in double precision (gradients: the taps' spectrum)
};

struct conv_args
{
    const void* in;    // channels x n samples
    void* out;
    const void* hist;  // channels x nhist previous samples
    long long n;       // samples per channel in this call
    long long nhist;   // M - 1
    long long m1;      // overlap of the blocks: M - 1, rounded up to even for unpaired blocks
    long long bo;      // valid outputs per block
    int channels;
    const void* hspec; // c+1 complex: FFT_F(taps) / F
    const void* rtw;   // W_F^k, k = 0..c
    const void* tw;
    conv_fft fft;      // c = F/2 point complex FFT
};

template <typename T>
cudaError_t launch_conv_os(const conv_args& a, long long nblocks, cudaStream_t st);

// k_fir_bwd: gradients of `blocks` blocks per channel.
struct fir_bwd_args
{
    const void* x;
    const void* grad_y;
    void* grad_x;  // may be null
    void* partial; // one spectrum of c + 1 values per CTA (null: no taps gradient)
    long long n, bo, blocks, channels;
    const void* hspec;
    const void* rtw;
    const void* tw;
    conv_fft fft;
    int elems; // shared complex elements of one block
};

// fir_backward (adjoint.hpp) block by block; false (nothing done) when the taps are too long for one CTA's FFT.
// Enqueued on st.
template <typename T>
bool fir_backward_blocks(const T* taps, long long ntaps, long long channels, long long n, const T* x, const T* grad_y,
                         T* grad_x, T* grad_h, cudaStream_t st);

template <typename T>
cudaError_t launch_hist_update(const void* hist_old, void* hist_new, const void* in, long long n, long long m1,
                               int channels, cudaStream_t st);

template <typename T>
class conv_filter
{
public:
    // taps: host or device pointer to `ntaps` values; block_size is the reference's partition size and
    // only bounds the blocks from below here (outputs do not depend on it but for rounding).  Taps too long for one
    // overlap-save FFT per CTA (M - 1 >= F / 2 at the largest one-CTA F) take the long mode: each call
    // convolves [history, input] with the taps through one real-FFT convolution per channel.
    conv_filter(const T* taps, size_t ntaps, size_t block_size, int channels = 1);
    // in / out: device pointers to channels x n samples (channel-major).  out must not alias in.
    void process(T* out, const T* in, size_t n, cudaStream_t st);
    void reset();
    size_t taps() const { return m_; }
    size_t fft_size() const { return f_; }
    int channels() const { return channels_; }
    bool long_mode() const { return long_; }
    int launches(size_t n) const;

private:
    size_t m_, f_, c_, bo_;
    int channels_;
    bool long_ = false;
    std::unique_ptr<fir_tables<T>> tables_;
    dbuf hspec_, hist_[2];
    dbuf htaps_, lin_, lout_; // long mode: taps, [history, input] and the full convolution of one channel
    int cur_ = 0;
};

} // namespace kfr_gpu
