// Plans of the runtime-length block FFT (rp_fft.cuh): radix choice, shared-memory layouts and launch shapes.
// Plain C++, shared by the host planner and the kernels.
//
// A length n = R_0 R_1 ... runs as self-sorting (Stockham) passes over a tile of `nsig` signals.  Butterfly j
// of pass p (stride ns = R_0 .. R_{p-1}, j = q ns + k) reads inputs j + r n / R and writes outputs
// q R ns + k + r ns.  Between two passes the tile sits in one shared buffer whose layout puts `pad` spare
// slots after every ns' = R_0 .. R_p elements: element i is at i + (i / ns') pad.  Because n / R of the next
// pass is a multiple of ns', both the stores of this pass and the loads of the next one are linear in r, so a
// butterfly computes two addresses and then steps by a constant; pads chosen per pass keep the strided
// stores free of bank conflicts.
#pragma once

#include <cstdint>
#include <vector>

namespace kfr_gpu
{

constexpr int kRpMaxPasses  = 8;
constexpr int kRpMaxRadix   = 16;

// Values a thread holds across the barrier of an in-place pass: 16, or 32 in half as many threads for lengths
// that 16 per thread cannot hold.
constexpr int kRpHold     = 16;
constexpr int kRpLongHold = 32;

// Threads of a CTA for complex values of `elem` bytes (64 registers per thread for complex<float> at 16 values
// held, 128 for complex<double>).
#if defined(__CUDACC__)
__host__ __device__
#endif
    constexpr int rp_max_threads(int elem, int hold)
{
    return (elem == 8 ? 1024 : 512) * kRpHold / hold;
}

struct rp_pass
{
    int radix, ns, nbf; // nbf = n / radix butterflies per signal
    uint32_t mq;        // j / ns = mulhi(j, mq) (0: ns == 1)
    uint32_t mg;        // J / nbf = mulhi(J, mg) for J over the tile's butterflies (0: nbf == 1)
    int fast;           // tile butterflies: 0: J = g nbf + j, 1: J = j S + g (signals fastest)
    // load of input r:   j ld_e + q ld_q + g ld_g + r ld_r  (not used by a first pass that reads global memory)
    int ld_e, ld_q, ld_g, ld_r;
    // store of output r: k st_e + q st_q + g st_g + r st_r  (not used by a last pass that writes global memory)
    int st_e, st_q, st_g, st_r;
    int tw_off;         // W_{ns R}^k, k < ns, at tw[tw_off + k]; row r - 1 at + (r - 1) ns
    int wr_off;         // radix above 16: W_R^m, m < R, at tw[wr_off + m]
};

struct rp_desc
{
    int n, npass;
    int shift; // fast layouts: log2 of the signals per tile
    int elems; // shared elements per signal (RP_SIGNALS) or per tile
    int hold;  // values a thread holds
    rp_pass pass[kRpMaxPasses];
};

// Butterflies of radix R a thread holds in registers across the barrier of an in-place pass (radices above 16,
// primes, hold `hold` outputs of any butterflies instead: see rp_threads_needed).
#if defined(__CUDACC__)
__host__ __device__
#endif
    constexpr int rp_held(int R, int hold)
{
    return hold / R;
}

// Order in which a tile's butterflies and signals are laid out.
enum rp_layout
{
    RP_SIGNALS, // contiguous signals: a signal's butterflies on consecutive threads
    RP_COLS,    // columns of a row-major array: the S columns of a tile on consecutive threads
    RP_ROWS,    // read as contiguous signals, written with the S signals on consecutive threads
};

// Radices of n in pass order for threads that hold `hold` values, empty when n has a prime factor above `largest` (13,
// or up to 127) or needs too many passes.  Primes above 13 run as in-place passes of dot products between codelet passes
// (of radix 1, a copy, where no other factor is left).
std::vector<int> rp_radices(long long n, int largest = 13, int hold = kRpHold);

// n as 16 16 .. 8, 4 or 2, then 9s, 3, 5s, 7s, 11s, 13s and the primes up to `largest`; empty if it has a larger one.
std::vector<int> rp_plain_radices(long long n, int largest);

// The cheapest radices whose passes all fit a CTA in place (rp_fits with smem_io), empty if none do.  Near the longest
// one-CTA lengths a thread has room for one butterfly of radix 9 to 15 only, so that the radices that would be fastest
// (rp_radices) need more threads than a CTA has.
std::vector<int> rp_radices_held(long long n, int largest, int elem, int smem_budget, int hold);

// Descriptor of the radices over a tile.  elem: bytes of a complex value; S (a power of two): signals per tile
// of RP_COLS and RP_ROWS.  smem_io: the first pass reads and the last pass writes shared memory too, element
// i of signal g at g n + i.
rp_desc rp_build(const std::vector<int>& radices, rp_layout layout, int S, int elem, bool smem_io = false,
                 int hold = kRpHold);

// Shared-memory elements per signal (RP_SIGNALS) or per tile of S signals (RP_COLS, RP_ROWS).
int rp_smem_elems(const rp_desc& d, rp_layout layout, int S, bool smem_io = false);

// Threads the in-place passes of `nsig` signals need (every butterfly held by some thread); 1 if there are none.
int rp_threads_needed(const rp_desc& d, int nsig, bool smem_io = false);

// Whether one signal of the radices fits a CTA of `smem_budget` bytes (an estimate that rp_choose confirms).
bool rp_fits(const std::vector<int>& radices, int elem, int smem_budget, bool smem_io = false, int hold = kRpHold);

// Launch shape for contiguous signals: signals per CTA and threads.
struct rp_shape
{
    int spc = 0, threads = 0; // spc 0: n does not fit one CTA
};
rp_shape rp_choose(const rp_desc& d, int sig_elems, int elem, int smem_budget, bool smem_io = false);
// The shape for a batch that gives few CTAs per SM: fewer signals per CTA.
rp_shape rp_shrink(const rp_desc& d, const rp_shape& full, long long batch, int sms, bool smem_io = false);

// Signals per tile of RP_COLS / RP_ROWS: 128-byte rows (16 complex<float>), wider for short signals so that a
// tile has work for a few warps, narrower where the threads or, with a sixteenth of padding, `smem_budget`
// bytes need it (0: none).
int rp_tile(const std::vector<int>& radices, int elem, int smem_budget, int hold = kRpHold);

// Relative cost per element of a radix-R pass (instructions, from the codelets' operation counts).
double rp_pass_cost(int R);

} // namespace kfr_gpu
