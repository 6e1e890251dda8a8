// Uneven batch: persistent dependency-aware work-queue kernel, plan, autotuner and graph capture
// (uneven.hpp).
#include "uneven.hpp"
#include "kernels.cuh"
#include "rp_fft.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <sstream>

namespace kfr_gpu
{

// ------------------------------------------------------------------------------------------------------
// kernel
// ------------------------------------------------------------------------------------------------------

__device__ __forceinline__ int ld_acquire(const int* p)
{
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// L2 load (bypasses L1): data another CTA wrote during this launch
__device__ __forceinline__ cpx<float> ld_cg(const cpx<float>* p)
{
    const float2 v = __ldcg(reinterpret_cast<const float2*>(p));
    return mk<float>(v.x, v.y);
}
__device__ __forceinline__ cpx<double> ld_cg(const cpx<double>* p)
{
    const double2 v = __ldcg(reinterpret_cast<const double2*>(p));
    return mk<double>(v.x, v.y);
}

// The persistent kernel on the runtime-length block FFT (rp_fft.cuh).  Every item is a tile of signals, columns
// or rows whose element i of signal g lies at base[g] + i stride, so one instance of the passes serves all
// of them; the first pass reads and the last pass writes global memory, with the chirps, the spectrum product
// and the four-step twiddle in its functors.  Four 256-thread CTAs per SM (64 registers; two of 512 threads
// for plans with passes longer than 4096 points), so that one's queue round trip, loads and barriers overlap
// with the others' arithmetic.  Bound by instruction issue and by the latency of an item's chain (queue, job,
// loads, barriers).  1024 signals of 64 to 65536 points: 186 us against 746 us for runtime passes of 690
// instructions per element in one 512-thread CTA per SM.
template <typename T>
__global__ void __launch_bounds__(kUnevenThreads, 2) k_uneven(const __grid_constant__ uneven_launch a)
{
    stream_order();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ rp_desc D;
    // input and output 0 of each signal of the tile, and its column / row
    __shared__ const cpx<T>* s_src[kUnevenMaxSpc];
    __shared__ cpx<T>* s_dst[kUnevenMaxSpc];
    __shared__ int s_col[kUnevenMaxSpc];
    // the last input and the first output index outside a Bluestein transform's signal
    __shared__ int s_ilim[kUnevenMaxSpc], s_olim[kUnevenMaxSpc];
    __shared__ uneven_job J;
    __shared__ uneven_item W;
    __shared__ int s_item, s_fft;
    cpx<T>* sm = reinterpret_cast<cpx<T>*>(smem_raw);
    const bool inv = a.inverse != 0;
    if (threadIdx.x == 0)
        s_fft = -1;
    for (;;)
    {
        __syncthreads();
        if (threadIdx.x == 0)
        {
            const int it = atomicAdd(a.queue, 1);
            s_item       = it;
            if (it < a.nitems)
            {
                W = a.items[it];
                J = a.jobs[W.job];
                if (J.wait >= 0)
                {
                    // every tile of the stage waited for was dequeued before this one and runs on a resident
                    // CTA, so the counter reaches `need`; the bound only guards against a fault elsewhere
                    uint32_t spins = 0;
                    while (ld_acquire(a.counters + J.wait) < J.need + a.stage_bias)
                    {
                        if (spins++ >= a.wait_spins)
                        {
                            atomicExch(a.err, 1); // carry on: the tile's loads stay inside its buffers
                            break;
                        }
                        __nanosleep(256);
                    }
                }
            }
        }
        __syncthreads();
        if (s_item >= a.nitems)
            break;
        const int mode = J.mode, cnt = W.count, first = W.first;
        const int n1 = J.n1, n2 = J.n2;
        if (J.fft != s_fft)
        {
            const int* src = reinterpret_cast<const int*>(&a.ffts[J.fft].d);
            for (int i = threadIdx.x; i < int(sizeof(rp_desc) / sizeof(int)); i += blockDim.x)
                reinterpret_cast<int*>(&D)[i] = src[i];
        }
        if (int(threadIdx.x) < cnt)
        {
            const cpx<T>* src = reinterpret_cast<const cpx<T>*>(J.src == 0 ? a.in : J.src == 1 ? a.out : a.scratch) + J.src_off;
            cpx<T>* dst       = reinterpret_cast<cpx<T>*>(J.dst == 2 ? a.scratch : a.out) + J.dst_off;
            const int g       = threadIdx.x;
            // columns and rows beyond the last repeat it: they read the same values and store the same results
            const int c = mode <= UM_BLUE1 ? 0 : min(first + g, (mode == UM_COL ? n2 : n1) - 1);
            const long long b = mode <= UM_BLUE1 ? a.offsets[first + g] : c;
            const int nv      = int(J.nvalid);
            s_src[g]          = src + (mode == UM_ROW ? (long long)c * n2 : J.pre ? min(c, nv - 1) : b);
            s_dst[g]          = dst + b;
            s_col[g]          = c;
            s_ilim[g]         = J.pre ? max(nv - 1 - c, 0) / n2 : 0x7fffffff;
            s_olim[g]         = J.post == 2 ? (max(nv - c, 0) + n1 - 1) / n1 : 0x7fffffff;
        }
        __syncthreads();
        if (threadIdx.x == 0)
            s_fft = J.fft;
        const cpx<T>* tw    = reinterpret_cast<const cpx<T>*>(a.ffts[J.fft].tw);
        const cpx<T>* chirp = reinterpret_cast<const cpx<T>*>(J.chirp);
        const cpx<T>* bhat  = reinterpret_cast<const cpx<T>*>(J.bhat);
        if (mode == UM_BLUE1)
        {
            // one-CTA Bluestein: both transforms from and to shared memory
            const int m = D.n, n = J.n;
            for (int i = threadIdx.x; i < cnt * m; i += blockDim.x)
            {
                const int g = i / m, e = i - g * m;
                sm[i]       = e < n ? conj_if(ld_cg(s_src[g] + e), inv) * ldg(chirp + e) : mk<T>(0, 0);
            }
            __syncthreads();
#pragma unroll 1
            for (int round = 0;; round++)
            {
                rp_run_smem<T>(D, sm, cnt, tw);
                if (round)
                    break;
                for (int i = threadIdx.x; i < cnt * m; i += blockDim.x)
                    sm[i] = conj(sm[i] * ldg(bhat + i % m));
                __syncthreads();
            }
            for (int i = threadIdx.x; i < cnt * n; i += blockDim.x)
            {
                const int g = i / n, e = i - g * n;
                s_dst[g][e] = conj_if(conj(sm[g * m + e]) * ldg(chirp + e), inv);
            }
        }
        else
        {
            const bool cin = J.first && inv, cout = J.last && inv;
            // bytes between a signal's input / output elements; elements between them
            const int is = mode == UM_COL ? n2 : 1, os = mode == UM_COL ? n2 : mode == UM_ROW ? n1 : 1;
            const uint32_t isb = uint32_t(is) * sizeof(cpx<T>), osb = uint32_t(os) * sizeof(cpx<T>);
            const int nv = int(J.nvalid), pre = J.pre, post = J.post;
            rp_run<T>(
                D, sm, cnt, tw,
                [&](int g, int i)
                {
                    // the zero padding repeats a column's last value (prep clears it)
                    return conj_if(ld_cg(rp_at(s_src[g], min(i, s_ilim[g]), isb)), cin);
                },
                [&](int g, int i, cpx<T> v)
                {
                    if (i < s_olim[g])
                        *rp_at(s_dst[g], i, osb) = conj_if(v, cout);
                },
                [&](int g, int k, int step, auto& o)
                {
                    constexpr int R = int(sizeof(o) / sizeof(o[0]));
                    const int col   = s_col[g];
                    if (post)
                    {
                        // 1: conj(v bhat), 2: conj(v) chirp, conjugated once more for the inverse
#pragma unroll
                        for (int r = 0; r < R; r++)
                        {
                            const int e = col + (k + r * step) * os;
                            if (post == 1)
                                o[r] = conj(o[r] * ldg(bhat + e));
                            else if (e < nv)
                                o[r] = conj(o[r]) * ldg(chirp + e);
                        }
                    }
                    if (mode != UM_COL)
                        return;
                    // four-step twiddle: W^{col k} times powers of the butterfly's step W^{col step}; col k and
                    // col step are below the length, at most 8192^2
                    const cpx<T>* twA = reinterpret_cast<const cpx<T>*>(J.twA);
                    const cpx<T>* twB = reinterpret_cast<const cpx<T>*>(J.twB);
                    const int lbits   = J.lbits, mask = (1 << lbits) - 1;
                    const auto root = [&](int m) { return ldg(twA + (m >> lbits)) * ldg(twB + (m & mask)); };
                    if constexpr (R >= 8)
                        twiddle_powers4<T, R>(o, root(col * step), root(4 * col * step));
                    else if constexpr (R > 1)
                        twiddle_powers<T, R>(o, root(col * step));
                    const cpx<T> w = root(col * k);
#pragma unroll
                    for (int r = 0; r < R; r++)
                        o[r] = o[r] * w;
                },
                [&](int g, int j, int step, auto& v)
                {
                    if (!pre)
                        return;
                    // Bluestein's chirp, zero beyond the signal
                    constexpr int R = int(sizeof(v) / sizeof(v[0]));
#pragma unroll
                    for (int r = 0; r < R; r++)
                    {
                        const int e = s_col[g] + (j + r * step) * is;
                        v[r]        = e < nv ? v[r] * ldg(chirp + e) : mk<T>(0, 0);
                    }
                });
        }
        __syncthreads();
        if (threadIdx.x == 0 && J.done >= 0)
        {
            __threadfence();
            atomicAdd(a.counters + J.done, 1);
        }
    }
}

cudaError_t launch_uneven_f32(const uneven_launch& a, int threads, int smem, int grid, cudaStream_t st)
{
    const cudaError_t e = prepare_launch(reinterpret_cast<const void*>(k_uneven<float>), threads, smem);
    if (e != cudaSuccess)
        return e;
    return launch_kernel(k_uneven<float>, dim3(unsigned(grid)), threads, size_t(smem), st, a);
}

// Dynamic shared memory of one of four 256-thread or two 512-thread CTAs per SM, beside the kernel's static
// descriptor, offsets and job.
static int uneven_smem(int threads) { return threads <= 256 ? 48 * 1024 : 104 * 1024; }

// ------------------------------------------------------------------------------------------------------
// plan
// ------------------------------------------------------------------------------------------------------

namespace
{

std::mutex g_tune_mu;
// threads per CTA and length -> fastest radix order and tile (measured in CTAs of that shape)
std::map<std::pair<int, long long>, std::pair<std::vector<int>, int>> g_tune;

// Descriptors that the plan being built on this thread has asked for: building one (10 us, mostly counting bank conflicts)
// for each question about a length made a plan of 4096 short signals take 49 ms instead of 12.
struct desc_memo
{
    std::map<std::tuple<std::vector<int>, int, int, bool>, rp_desc> known;
    desc_memo* const outer;
    static thread_local desc_memo* current;
    desc_memo() : outer(current) { current = this; }
    ~desc_memo() { current = outer; }
};
thread_local desc_memo* desc_memo::current = nullptr;

// descriptor of a one-CTA transform, or of a tile of S columns / rows; false if it does not fit a CTA
bool fits(int threads, const std::vector<int>& order, rp_layout layout, int S, bool smem_io, rp_desc& d, int& elems)
{
    if (order.empty())
        return false;
    if (desc_memo* memo = desc_memo::current)
    {
        const auto key = std::make_tuple(order, int(layout), S, smem_io);
        auto f         = memo->known.find(key);
        if (f == memo->known.end())
            f = memo->known.emplace(key, rp_build(order, layout, S, 8, smem_io)).first;
        d = f->second;
    }
    else
        d = rp_build(order, layout, S, 8, smem_io);
    elems = rp_smem_elems(d, layout, S, smem_io);
    return rp_threads_needed(d, S, smem_io) <= threads && elems * 8 <= uneven_smem(threads);
}

std::vector<int> radices_of(long long m)
{
    return m == 1 ? std::vector<int>{ 1 } : rp_radices(m, kGenericMax);
}

bool fits_one_cta(int threads, long long m, const std::vector<int>& order, bool smem_io)
{
    rp_desc d;
    int elems = 0;
    return m <= threads * kRpMaxRadix && fits(threads, order, RP_SIGNALS, 1, smem_io, d, elems);
}

// most signals of one item: about 16 values per thread, every in-place butterfly held
int most_signals(int threads, const rp_desc& d, int elems, bool smem_io)
{
    int spc = std::max(1, std::min({ threads * kRpMaxRadix / std::max(1, d.n), uneven_smem(threads) / (elems * 8),
                                     kUnevenMaxSpc }));
    while (spc > 1 && rp_threads_needed(d, spc, smem_io) > threads)
        spc--;
    return spc;
}

std::vector<std::vector<int>> candidate_orders(long long m)
{
    std::vector<std::vector<int>> c;
    const auto a = radices_of(m);
    if (a.empty())
        return c;
    auto add = [&](std::vector<int> v)
    {
        // the ends are codelets
        if (v.front() <= kRpMaxRadix && v.back() <= kRpMaxRadix && std::find(c.begin(), c.end(), v) == c.end())
            c.push_back(v);
    };
    add(a);
    add(std::vector<int>(a.rbegin(), a.rend()));
    auto d = a;
    std::sort(d.begin(), d.end(), std::greater<int>());
    add(d);
    std::sort(d.begin(), d.end());
    add(d);
    return c;
}

// Columns / rows of an m-point FFT per item: the largest power of two of about 16 values per thread that fits
// (an item costs a queue round trip and a few barriers whatever its size), 0 if none.
int tile_of(int threads, const std::vector<int>& order, rp_layout layout)
{
    rp_desc d;
    int elems   = 0;
    long long m = 1;
    for (int r : order)
        m *= r;
    for (int S = kUnevenMaxSpc; S >= 1; S /= 2)
        if (S * m <= threads * kRpMaxRadix && fits(threads, order, layout, S, false, d, elems))
            return S;
    return 0;
}

// four-step split n = n1 * n2 with the cheapest passes (rows of fewer than 16 columns cost extra sectors)
struct splitter
{
    int threads;
    std::map<std::pair<long long, int>, double> memo;
    std::map<long long, double> least_memo;
    // the least that cost(m) can be, from the radices and the tile's largest size alone; -1 if there is no tile
    double least(long long m)
    {
        auto f = least_memo.find(m);
        if (f != least_memo.end())
            return f->second;
        const auto rad = radices_of(m);
        int S          = 16;
        while (S > 1 && S * m > threads * kRpMaxRadix)
            S /= 2;
        double c = rad.empty() ? -1 : 12.0 * (16.0 / S - 1);
        for (int r : rad)
            c += rp_pass_cost(r);
        return least_memo[m] = c;
    }
    double cost(long long m, rp_layout layout)
    {
        const auto key = std::make_pair(m, int(layout));
        auto f         = memo.find(key);
        if (f != memo.end())
            return f->second;
        double c       = -1;
        const auto rad = radices_of(m);
        const int S    = rad.empty() ? 0 : tile_of(threads, rad, layout);
        if (S)
        {
            c = 12.0 * (16.0 / std::min(S, 16) - 1);
            for (int r : rad)
                c += rp_pass_cost(r);
        }
        return memo[key] = c;
    }
    bool split(long long n, int& n1, int& n2)
    {
        double best       = -1;
        const long long t = (long long)threads * kRpMaxRadix;
        // the cost of the most balanced split: planning the tiles of those that cannot reach it takes milliseconds
        double bound = 1e30;
        for (long long a = (long long)std::sqrt(double(n)); a >= 2 && n / a <= t; a--)
            if (n % a == 0)
            {
                const double c = cost(a, RP_COLS), r = cost(n / a, RP_ROWS);
                if (c >= 0 && r >= 0)
                    bound = c + r;
                break;
            }
        for (long long a = 2; a <= t && a * 2 <= n; a++)
        {
            if (n % a || n / a > t)
                continue;
            const double la = least(a), lb = least(n / a);
            if (la < 0 || lb < 0 || la + lb > (best >= 0 ? std::min(best, bound) : bound) + 1e-6)
                continue;
            const double c = cost(a, RP_COLS), r = c < 0 ? -1 : cost(n / a, RP_ROWS);
            // of equal splits the most balanced
            if (r >= 0 && (best < 0 || c + r < best - 1e-9 ||
                           (c + r < best + 1e-9 && std::max(a, n / a) < std::max(n1, n2))))
            {
                best = c + r;
                n1   = int(a);
                n2   = int(n / a);
            }
        }
        return best >= 0;
    }
};

// Convolution length of a Bluestein transform: the smallest power of two >= 2n - 1.
long long bluestein_length(long long n)
{
    long long m = 1;
    while (m < 2 * n - 1)
        m <<= 1;
    return m;
}

} // namespace

int uneven_plan::get_shape(long long m, int layout, int S, bool smem_io)
{
    const shape_key key(m, layout, S, smem_io);
    auto f = shape_of_.find(key);
    if (f != shape_of_.end())
        return f->second;
    std::vector<int> o = radices_of(m);
    if (layout == RP_SIGNALS && !smem_io)
    {
        std::lock_guard<std::mutex> g(g_tune_mu);
        auto t = g_tune.find({ threads_, m });
        rp_desc d;
        int elems = 0;
        if (t != g_tune.end() && fits(threads_, t->second.first, RP_SIGNALS, 1, false, d, elems))
            o = t->second.first;
    }
    shape s;
    if (!fits(threads_, o, rp_layout(layout), S, smem_io, s.d, s.elems))
        throw std::invalid_argument("internal: uneven batch shape exceeds one CTA");
    // one twiddle table per radix order
    auto t = tw_of_.find(o);
    if (t == tw_of_.end())
    {
        const auto table = pass_twiddles<float>(o); 
        tables_.emplace_back(new dbuf);
        tables_.back()->upload(table.data(), table.size() * sizeof(table[0]));
        t = tw_of_.emplace(o, tables_.back()->get()).first;
    }
    s.tw          = t->second;
    const int idx = int(shapes_.size());
    shapes_.push_back(s);
    shape_of_[key] = idx;
    return idx;
}

uneven_plan::uneven_plan(const std::vector<long long>& lengths, bool autotune) : lengths_(lengths)
{
    offsets_.resize(lengths.size());
    for (size_t i = 0; i < lengths.size(); i++)
    {
        if (lengths[i] < 1)
            throw std::invalid_argument("every signal length must be at least 1");
        offsets_[i] = total_;
        total_ += lengths[i];
    }
    check(cudaStreamCreateWithFlags(&cap_, cudaStreamNonBlocking), "create stream");
    err_.alloc();
    desc_memo memo;
    std::vector<long long> distinct(lengths);
    std::sort(distinct.begin(), distinct.end());
    distinct.erase(std::unique(distinct.begin(), distinct.end()), distinct.end());

    // 256-thread CTAs, four per SM; 512-thread CTAs, two per SM, where a length needs passes that only they can hold, or
    // where the longest transforms are of 4097 to 8192 points, so that every signal is one item then.  Signals of up to
    // 4096 points (Bluestein convolutions of 8192), 200 / 1024 of them: 35 / 42 us with 256 threads, 28 / 37 with 512; up
    // to 2048 points (convolutions of 4096), 1024 of them: 23 and 25.5; up to 65536 points, 1024 of them: 161 and 164.
    const auto plannable = [&](splitter& sp, long long n)
    {
        const bool smooth = is_smooth(n);
        const long long m = smooth ? n : bluestein_length(n);
        int n1 = 0, n2 = 0;
        return fits_one_cta(sp.threads, m, radices_of(m), !smooth) || sp.split(m, n1, n2);
    };
    long long longest   = 0;
    const auto one_item = [&](long long n)
    {
        const bool smooth = is_smooth(n);
        const long long m = smooth ? n : bluestein_length(n);
        longest           = std::max(longest, m);
        return fits_one_cta(kUnevenThreads, m, radices_of(m), !smooth);
    };
    splitter splits{ 256, {} };
    if ((std::all_of(distinct.begin(), distinct.end(), one_item) && longest > 4096) ||
        !std::all_of(distinct.begin(), distinct.end(), [&](long long n) { return plannable(splits, n); }))
        splits = splitter{ kUnevenThreads, {} };
    threads_ = splits.threads;
    int dev = 0, sms = 152;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);

    // autotuner for the one-CTA lengths present: time candidate radix orders and tiles on a synthetic batch
    // of that length alone, keep the fastest for the process
    if (autotune)
    {
        std::vector<long long> todo;
        for (long long n : distinct)
            if (n > 1 && fits_one_cta(threads_, n, radices_of(n), false))
                todo.push_back(n);
        dbuf tin, tout, tffts, tjobs, titems, toffs, tq, ttw;
        const long long tune_elems = 1 << 20;
        tin.alloc(size_t(tune_elems) * 8);
        tout.alloc(size_t(tune_elems) * 8);
        check(cudaMemset(tin.get(), 0, tin.size()), "clear tuning input");
        tq.alloc(sizeof(int));
        cudaEvent_t e0, e1;
        check(cudaEventCreate(&e0), "event");
        check(cudaEventCreate(&e1), "event");
        for (long long n : todo)
        {
            {
                std::lock_guard<std::mutex> g(g_tune_mu);
                if (g_tune.count({ threads_, n }))
                    continue;
            }
            float best = 1e30f;
            std::pair<std::vector<int>, int> best_cfg(radices_of(n), 0);
            for (const auto& order : candidate_orders(n))
            {
                uneven_fft f{};
                int elems = 0;
                if (!fits(threads_, order, RP_SIGNALS, 1, false, f.d, elems))
                    continue;
                const auto table = pass_twiddles<float>(order);
                ttw.upload(table.data(), table.size() * sizeof(table[0]));
                f.tw           = ttw.get();
                const int smax = most_signals(threads_, f.d, elems, false);
                for (int spc : { smax, std::max(1, smax / 2) })
                {
                    const long long nsig = std::max<long long>(spc, std::min<long long>(4096, tune_elems / n));
                    std::vector<long long> offs(nsig);
                    for (long long s = 0; s < nsig; s++)
                        offs[s] = s * n;
                    std::vector<uneven_item> its;
                    for (long long s = 0; s < nsig; s += spc)
                        its.push_back({ 0, int(s), int(std::min<long long>(spc, nsig - s)) });
                    uneven_job j{};
                    j.mode = UM_DIRECT;
                    j.dst  = 1;
                    j.fft  = 0;
                    j.n    = int(n);
                    j.wait = -1;
                    j.done = -1;
                    tffts.upload(&f, sizeof(f));
                    tjobs.upload(&j, sizeof(j));
                    titems.upload(its.data(), its.size() * sizeof(uneven_item));
                    toffs.upload(offs.data(), offs.size() * sizeof(long long));
                    uneven_launch L{ static_cast<uneven_fft*>(tffts.get()), static_cast<uneven_job*>(tjobs.get()),
                                     static_cast<uneven_item*>(titems.get()), static_cast<long long*>(toffs.get()),
                                     int(its.size()), static_cast<int*>(tq.get()), nullptr,
                                     err_.get(), tin.get(), tout.get(), nullptr, 0 };
                    const int smem = spc * elems * 8;
                    const int grid = std::min<int>(int(its.size()), 1024 / threads_ * sms);
                    for (int rep = 0; rep < 4; rep++)
                    {
                        check(cudaMemset(tq.get(), 0, sizeof(int)), "clear queue");
                        if (rep == 1)
                            check(cudaEventRecord(e0), "event");
                        check(launch_uneven_f32(L, threads_, smem, grid, nullptr), "tune");
                    }
                    float ms = 0;
                    check(cudaEventRecord(e1), "event");
                    check(cudaEventSynchronize(e1), "tune");
                    check(cudaEventElapsedTime(&ms, e0, e1), "tune");
                    if (ms / float(nsig) < best)
                    {
                        best     = ms / float(nsig);
                        best_cfg = { order, spc };
                    }
                }
            }
            std::lock_guard<std::mutex> g(g_tune_mu);
            g_tune[{ threads_, n }] = best_cfg;
        }
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
    }

    // jobs and items.  Stage s of every signal is listed after all of stage s-1 (stage 0: whole signals and
    // first column passes), each stage heaviest first.
    std::vector<uneven_job> jobs;
    std::vector<std::vector<uneven_item>> stage_items(4);
    std::vector<std::vector<double>> stage_cost(4);
    std::vector<long long> offs;
    long long scratch_elems = 0;
    auto add_item = [&](int stage, const uneven_item& it, double cost)
    {
        stage_items[stage].push_back(it);
        stage_cost[stage].push_back(cost);
    };
    auto tables = [&]() -> dbuf&
    {
        tables_.emplace_back(new dbuf);
        return *tables_.back();
    };
    // one-CTA lengths: a job per length over its signals
    std::map<long long, std::vector<int>> by_len;
    for (size_t i = 0; i < lengths.size(); i++)
        by_len[lengths[i]].push_back(int(i));
    for (auto& kv : by_len)
    {
        const long long n = kv.first;
        const auto& sig   = kv.second;
        const bool smooth = is_smooth(n);
        const bool direct = smooth && fits_one_cta(threads_, n, radices_of(n), false);
        long long m       = n;
        if (!smooth)
            m = bluestein_length(n);
        if (direct || (!smooth && fits_one_cta(threads_, m, radices_of(m), true)))
        {
            uneven_job j{};
            j.mode  = direct ? UM_DIRECT : UM_BLUE1;
            j.dst   = 1;
            j.first = j.last = 1;
            j.fft   = get_shape(m, RP_SIGNALS, 1, !direct);
            j.n     = int(n);
            j.wait  = -1;
            j.done  = -1;
            if (!direct)
            {
                dbuf& ch = tables();
                dbuf& bh = tables();
                bluestein_tables<float>(n, m, ch, bh);
                j.chirp = ch.get();
                j.bhat  = bh.get();
                n_blue1_ += int(sig.size());
            }
            else
                n_direct_ += int(sig.size());
            const shape& sh = shapes_[j.fft];
            int spc         = most_signals(threads_, sh.d, sh.elems, !direct);
            if (direct)
            {
                std::lock_guard<std::mutex> g(g_tune_mu);
                auto f = g_tune.find({ threads_, m });
                if (f != g_tune.end() && f->second.second > 0)
                    spc = std::min(spc, f->second.second);
            }
            const int jid   = int(jobs.size());
            jobs.push_back(j);
            const int first = int(offs.size());
            for (int i : sig)
                offs.push_back(offsets_[i]);
            for (int s = 0; s < int(sig.size()); s += spc)
            {
                const int c = std::min(spc, int(sig.size()) - s);
                add_item(0, { jid, first + s, c }, double(c) * double(m) * std::log2(double(std::max<long long>(m, 2))) *
                                                       (direct ? 1.0 : 2.0));
            }
            smem_ = std::max(smem_, spc * sh.elems * 8);
            continue;
        }
        // long signals: four-step (smooth lengths) or four-step Bluestein (a large prime factor), per signal
        const bool blue = !smooth;
        int n1 = 0, n2 = 0;
        if (!splits.split(m, n1, n2))
            throw std::invalid_argument("uneven batch: length " + std::to_string(n) + " is not supported");
        const int S1 = tile_of(threads_, radices_of(n1), RP_COLS), S2 = tile_of(threads_, radices_of(n2), RP_ROWS);
        const int f1 = get_shape(n1, RP_COLS, S1, false), f2 = get_shape(n2, RP_ROWS, S2, false);
        smem_        = std::max({ smem_, shapes_[f1].elems * 8, shapes_[f2].elems * 8 });
        // W_m^k two-level table
        int lb = 0;
        while ((1LL << (2 * lb)) < m)
            lb++;
        const long long nb = 1LL << lb, na = (m + nb - 1) / nb;
        std::vector<std::complex<float>> A(na), B(nb);
        for (long long i = 0; i < na; i++)
        {
            const auto w = twiddle(i * nb, m);
            A[i]         = { float(w.real()), float(w.imag()) };
        }
        for (long long i = 0; i < nb; i++)
        {
            const auto w = twiddle(i, m);
            B[i]         = { float(w.real()), float(w.imag()) };
        }
        dbuf& tA = tables();
        dbuf& tB = tables();
        tA.upload(A.data(), A.size() * sizeof(A[0]));
        tB.upload(B.data(), B.size() * sizeof(B[0]));
        const void *chirp = nullptr, *bhat = nullptr;
        if (blue)
        {
            dbuf& ch = tables();
            dbuf& bh = tables();
            bluestein_tables<float>(n, m, ch, bh);
            chirp = ch.get();
            bhat  = bh.get();
        }
        const int ncol = (n2 + S1 - 1) / S1, nrow = (n1 + S2 - 1) / S2;
        const double c1 = double(S1) * n1 * std::log2(double(n1)), c2 = double(S2) * n2 * std::log2(double(n2));
        for (int i : sig)
        {
            const int base = ncounters_;
            ncounters_ += blue ? 3 : 1;
            const long long sc = scratch_elems;
            scratch_elems += blue ? 2 * m : m;
            auto stage_job = [&](int mode, int src, long long soff, int dst, long long doff, int pre, int post,
                                 bool first, bool last, int wait, int need, int done)
            {
                uneven_job j{};
                j.mode    = mode;
                j.fft     = mode == UM_COL ? f1 : f2;
                j.n       = mode == UM_COL ? n1 : n2;
                j.n1      = n1;
                j.n2      = n2;
                j.src     = src;
                j.dst     = dst;
                j.src_off = soff;
                j.dst_off = doff;
                j.pre     = pre;
                j.post    = post;
                j.first   = first;
                j.last    = last;
                j.nvalid  = n;
                j.chirp   = chirp;
                j.bhat    = bhat;
                j.twA     = tA.get();
                j.twB     = tB.get();
                j.lbits   = lb;
                j.wait    = wait;
                j.need    = need;
                j.done    = done;
                jobs.push_back(j);
                return int(jobs.size()) - 1;
            };
            const long long off = offsets_[i];
            if (!blue)
            {
                const int jc = stage_job(UM_COL, 0, off, 2, sc, 0, 0, true, false, -1, 0, base);
                const int jr = stage_job(UM_ROW, 2, sc, 1, off, 0, 0, false, true, base, ncol, -1);
                for (int c = 0; c < ncol; c++)
                    add_item(0, { jc, c * S1, S1 }, c1);
                for (int r = 0; r < nrow; r++)
                    add_item(1, { jr, r * S2, S2 }, c2);
                n_fourstep_++;
            }
            else
            {
                // convolution: (x chirp) -> FFT_m -> conj(. bhat) -> FFT_m -> conj(.) chirp, in four stages
                const int j0 = stage_job(UM_COL, 0, off, 2, sc, 1, 0, true, false, -1, 0, base);
                const int j1 = stage_job(UM_ROW, 2, sc, 2, sc + m, 0, 1, false, false, base, ncol, base + 1);
                const int j2 = stage_job(UM_COL, 2, sc + m, 2, sc, 0, 0, false, false, base + 1, nrow, base + 2);
                const int j3 = stage_job(UM_ROW, 2, sc, 1, off, 0, 2, false, true, base + 2, ncol, -1);
                for (int c = 0; c < ncol; c++)
                {
                    add_item(0, { j0, c * S1, S1 }, c1);
                    add_item(2, { j2, c * S1, S1 }, c1);
                }
                for (int r = 0; r < nrow; r++)
                {
                    add_item(1, { j1, r * S2, S2 }, c2);
                    add_item(3, { j3, r * S2, S2 }, c2);
                }
                n_blue_fs_++;
            }
        }
    }
    std::vector<uneven_item> items;
    for (int s = 0; s < 4; s++)
    {
        std::vector<size_t> idx(stage_items[s].size());
        for (size_t i = 0; i < idx.size(); i++)
            idx[i] = i;
        std::stable_sort(idx.begin(), idx.end(),
                         [&](size_t x, size_t y) { return stage_cost[s][x] > stage_cost[s][y]; });
        for (size_t i : idx)
            items.push_back(stage_items[s][i]);
    }
    nitems_ = int(items.size());
    std::vector<uneven_fft> ffts;
    for (const shape& sp : shapes_)
        ffts.push_back({ sp.d, sp.tw });
    if (!ffts.empty())
        dffts_.upload(ffts.data(), ffts.size() * sizeof(uneven_fft));
    if (!jobs.empty())
        djobs_.upload(jobs.data(), jobs.size() * sizeof(uneven_job));
    if (!items.empty())
        ditems_.upload(items.data(), items.size() * sizeof(uneven_item));
    if (!offs.empty())
        doffsets_.upload(offs.data(), offs.size() * sizeof(long long));
    dqueue_.alloc(sizeof(int));
    dcounters_.alloc(size_t(std::max(1, ncounters_)) * sizeof(int));
    if (scratch_elems)
        scratch_.alloc(size_t(scratch_elems) * 8);
    smem_ = std::max(smem_, 1024);
    grid_ = std::max(1, std::min(nitems_, 1024 / threads_ * sms));
}

uneven_plan::~uneven_plan()
{
    if (gexec_)
        cudaGraphExecDestroy(gexec_);
    if (cap_)
        cudaStreamDestroy(cap_);
}

void uneven_plan::enqueue(void* out, const void* in, bool inverse, cudaStream_t st)
{
    if (!nitems_)
        return;
    check(cudaMemsetAsync(dqueue_.get(), 0, sizeof(int), st), "clear work queue");
    if (ncounters_)
        check(cudaMemsetAsync(dcounters_.get(), 0, size_t(ncounters_) * sizeof(int), st), "clear stage counters");
    uneven_launch L{ static_cast<uneven_fft*>(dffts_.get()), static_cast<uneven_job*>(djobs_.get()),
                     static_cast<uneven_item*>(ditems_.get()), static_cast<long long*>(doffsets_.get()), nitems_,
                     static_cast<int*>(dqueue_.get()), static_cast<int*>(dcounters_.get()),
                     err_.get(), in, out, scratch_.get(), inverse ? 1 : 0, wait_limit(),
                     unreachable_ ? 1 : 0 };
    check(launch_uneven_f32(L, threads_, smem_, grid_, st), "launch uneven batch");
}

void uneven_plan::execute(void* out, const void* in, bool inverse, cudaStream_t st)
{
    if (!gexec_ || gin_ != in || gout_ != out || ginv_ != inverse || gspins_ != wait_limit() ||
        gunreach_ != unreachable_)
    {
        if (gexec_)
        {
            cudaGraphExecDestroy(gexec_);
            gexec_ = nullptr;
        }
        // the kernel's attributes are set outside the capture by one eager run
        enqueue(out, in, inverse, cap_);
        check(cudaStreamSynchronize(cap_), "uneven batch");
        cudaGraph_t g = nullptr;
        check(cudaStreamBeginCapture(cap_, cudaStreamCaptureModeThreadLocal), "begin capture");
        try
        {
            enqueue(out, in, inverse, cap_);
        }
        catch (...)
        {
            cudaStreamEndCapture(cap_, &g);
            if (g)
                cudaGraphDestroy(g);
            throw;
        }
        check(cudaStreamEndCapture(cap_, &g), "end capture");
        const cudaError_t e = cudaGraphInstantiate(&gexec_, g, 0);
        cudaGraphDestroy(g);
        check(e, "instantiate graph");
        gin_      = in;
        gout_     = out;
        ginv_     = inverse;
        gspins_   = wait_limit();
        gunreach_ = unreachable_;
    }
    check(cudaGraphLaunch(gexec_, st), "launch graph");
}

void uneven_plan::check_device_error() const
{
    if (err_.take())
        throw cuda_error("an uneven-batch tile gave up waiting for the stage it depends on (device error flag)");
}

void uneven_plan::execute_per_signal(void* out, const void* in, bool inverse, cudaStream_t st)
{
    // the plain form: a regular plan per distinct length, one execution per signal
    for (size_t i = 0; i < lengths_.size(); i++)
    {
        const long long n = lengths_[i];
        auto f            = engines_.find(n);
        if (f == engines_.end())
            f = engines_.emplace(n, std::unique_ptr<complex_engine<float>>(new complex_engine<float>(n))).first;
        const long long need = f->second->scratch_elems(1);
        if (need * 8 > (long long)plain_scratch_.size())
        {
            check(cudaStreamSynchronize(st), "plain form");
            plain_scratch_.alloc(size_t(need) * 8);
        }
        f->second->execute(static_cast<char*>(out) + offsets_[i] * 8, static_cast<const char*>(in) + offsets_[i] * 8, 1,
                           n, n, inverse, plain_scratch_.get(), st);
    }
}

std::string uneven_plan::describe() const
{
    std::ostringstream s;
    s << "uneven batch: " << lengths_.size() << " signals in " << nitems_ << " work items on " << grid_
      << " persistent CTAs (" << n_direct_ << " one-CTA, " << n_blue1_ << " one-CTA Bluestein, " << n_fourstep_
      << " four-step, " << n_blue_fs_ << " four-step Bluestein)";
    return s.str();
}

} // namespace kfr_gpu
