// Planner of the runtime-length block FFT (see rp.hpp).
#include "rp.hpp"

#include <algorithm>
#include <cstring>
#include <set>

namespace kfr_gpu
{

double rp_pass_cost(int R)
{
    // real operations of the codelet per element, plus shared loads and stores, addresses, twiddle and its
    // powers (11), the barrier (3) and the index arithmetic of a butterfly (25 instructions)
    double ops;
    if (R > kRpMaxRadix)
        return 14 + 8.0 * R; // a dot product of R terms per output
    switch (R)
    {
    case 1: ops = 0; break;
    case 2: ops = 2; break;
    case 3: ops = 5.3; break;
    case 4: ops = 4; break;
    case 5: ops = 8; break;
    case 6: ops = 7.3; break;
    case 7: ops = 9.5; break;
    case 8: ops = 8; break;
    case 9: ops = 12.4; break;
    case 10: ops = 9.2; break;
    case 11: ops = 13.6; break;
    case 12: ops = 9.3; break;
    case 13: ops = 15.7; break;
    case 14: ops = 11.4; break;
    case 15: ops = 12.5; break;
    default: ops = 11; break;
    }
    return ops + 14 + 25.0 / R;
}

namespace
{

// Calls go_fn(multiset, cost) for the multisets of codelet radices <= `top` with product n (descending) whose pass
// costs stay below `bound`, which go_fn may lower.
template <class G>
void splits(long long n, int top, double cost, std::vector<int>& cur, const double& bound, const G& go_fn)
{
    if (n == 1)
    {
        go_fn(cur, cost);
        return;
    }
    if (int(cur.size()) >= kRpMaxPasses)
        return;
    for (int r = int(std::min<long long>(top, n)); r >= 2; r--)
        if (n % r == 0 && cost + rp_pass_cost(r) < bound)
        {
            cur.push_back(r);
            splits(n / r, r, cost + rp_pass_cost(r), cur, bound, go_fn);
            cur.pop_back();
        }
}

// The largest radices in the middle (the in-place passes hold whole butterflies in registers, so their radix
// bounds the threads a tile needs), the smallest last.
std::vector<int> pass_order(const std::vector<int>& desc)
{
    if (desc.size() < 3)
        return desc;
    const size_t mid = desc.size() - 2;
    std::vector<int> o(desc);
    o[0] = desc[mid];
    for (size_t i = 0; i < mid; i++)
        o[i + 1] = desc[i];
    return o;
}

uint32_t magic(int d) { return d <= 1 ? 0u : uint32_t((uint64_t(1) << 32) / uint32_t(d) + 1); }

// Wavefronts beyond the minimum of one warp-wide shared access with the given lane addresses (elements of
// `elem` bytes): 128 bytes are served at a time, so lanes go 128 / elem at a time.
int conflicts(const int* addr, int lanes, int elem)
{
    const int per = 128 / elem;
    int extra     = 0;
    for (int b = 0; b < lanes; b += per)
    {
        const int e = std::min(lanes, b + per);
        int count[16] = {}, worst = 1;
        for (int i = b; i < e; i++)
        {
            const int bank = addr[i] % per;
            bool dup       = false;
            for (int h = b; count[bank] && h < i && !dup; h++)
                dup = addr[h] == addr[i];
            if (!dup)
                worst = std::max(worst, ++count[bank]);
        }
        extra += worst - 1;
    }
    return extra;
}

struct lane_map
{
    int g, j;
};
lane_map map_lane(int J, const rp_pass& p, int shift)
{
    if (p.fast)
        return { J & ((1 << shift) - 1), J >> shift };
    return { J / p.nbf, J % p.nbf };
}

int store_conflicts(const rp_pass& p, int shift, int elem, int first, int total)
{
    int a[32], n = 0;
    for (int J = first; J < std::min(first + 32, total); J++)
    {
        const lane_map m = map_lane(J, p, shift);
        const int q = m.j / p.ns, k = m.j - q * p.ns;
        a[n++] = k * p.st_e + q * p.st_q + m.g * p.st_g;
    }
    return n ? conflicts(a, n, elem) : 0;
}
int load_conflicts(const rp_pass& p, int shift, int elem, int first, int total)
{
    int a[32], n = 0;
    for (int J = first; J < std::min(first + 32, total); J++)
    {
        const lane_map m = map_lane(J, p, shift);
        const int q = m.j / p.ns;
        a[n++] = m.j * p.ld_e + q * p.ld_q + m.g * p.ld_g;
    }
    return n ? conflicts(a, n, elem) : 0;
}

// The layout after pass i (and before pass i + 1): `pad` slots after every ns' elements.
void set_layout(rp_desc& d, int i, int S, bool fast_layout, int pad)
{
    rp_pass& a   = d.pass[i];
    rp_pass& b   = d.pass[i + 1];
    const int e  = fast_layout ? S : 1;
    const int nn = a.ns * a.radix; // ns'
    const int sg = fast_layout ? 1 : d.n + d.n / nn * pad;
    a.st_e = e;
    a.st_q = nn * e + pad;
    a.st_g = sg;
    a.st_r = a.ns * e;
    b.ld_e = e;
    b.ld_q = pad;
    b.ld_g = sg;
    b.ld_r = b.nbf * e + b.nbf / nn * pad;
}

} // namespace

// Takes the primes of 17 to `largest` out of n.
static std::vector<int> take_primes(long long& n, int largest)
{
    std::vector<int> primes;
    for (int p : { 17, 19, 23, 29, 31, 37, 41, 43, 47, 53, 59, 61, 67, 71, 73, 79, 83, 89, 97, 101, 103, 107, 109, 113, 127 })
        while (p <= largest && n % p == 0)
        {
            primes.push_back(p);
            n /= p;
        }
    return primes;
}

// The codelet radices r with the primes between their ends (of radix 1, a copy, where there are fewer than two), empty
// if those are too many passes.
static std::vector<int> with_primes(std::vector<int> r, const std::vector<int>& primes)
{
    if (primes.empty())
        return r;
    while (r.size() < 2)
        r.push_back(1);
    r.insert(r.begin() + 1, primes.begin(), primes.end());
    return r.size() > size_t(kRpMaxPasses) ? std::vector<int>{} : r;
}

std::vector<int> rp_radices(long long n, int largest, int hold)
{
    if (n < 2 || n > (1 << 16))
        return {};
    std::vector<int> r;
    const auto primes = take_primes(n, largest);
    std::vector<int> cur;
    double best = 1e30;
    splits(n, kRpMaxRadix, 0, cur, best,
           [&](const std::vector<int>& s, double c)
           {
               const auto o = pass_order(s);
               for (size_t i = 1; primes.empty() && i + 1 < o.size(); i++)
               {
                   // more threads than the largest CTA (or its half, for two of them per SM) to hold a middle pass
                   const long long t = (n / o[i] + rp_held(o[i], hold) - 1) / rp_held(o[i], hold);
                   const int most    = rp_max_threads(8, hold);
                   c += t > most ? 1000 : t > most / 2 ? 4 : 0;
               }
               if (c < best)
               {
                   best = c;
                   r    = o;
               }
           });
    return best >= 1e30 ? std::vector<int>{} : with_primes(r, primes);
}

std::vector<int> rp_plain_radices(long long n, int largest)
{
    std::vector<int> r;
    for (int p : { 16, 8, 4, 2, 9, 3, 5, 7, 11, 13 })
        for (; n > 1 && n % p == 0; n /= p)
            r.push_back(p);
    for (int p : take_primes(n, largest))
        r.push_back(p);
    return n == 1 ? r : std::vector<int>{};
}

std::vector<int> rp_radices_held(long long n, int largest, int elem, int smem_budget, int hold)
{
    if (n < 2 || n > (1 << 16))
        return {};
    std::vector<int> r;
    const auto primes = take_primes(n, largest);
    std::vector<int> cur;
    double best = 1e30;
    splits(n, kRpMaxRadix, 0, cur, best,
           [&](const std::vector<int>& s, double c)
           {
               const auto o = with_primes(pass_order(s), primes);
               if (c < best && rp_fits(o, elem, smem_budget, true, hold))
               {
                   best = c;
                   r    = o;
               }
           });
    return r;
}

rp_desc rp_build(const std::vector<int>& radices, rp_layout layout, int S, int elem, bool smem_io, int hold)
{
    rp_desc d;
    std::memset(&d, 0, sizeof(d));
    d.npass = int(radices.size());
    d.hold  = hold;
    d.n     = 1;
    for (int r : radices)
        d.n *= r;
    while ((1 << d.shift) < S)
        d.shift++;
    int ns = 1, off = 0;
    for (int i = 0; i < d.npass; i++)
    {
        rp_pass& p = d.pass[i];
        p.radix    = radices[i];
        p.ns       = ns;
        p.nbf      = d.n / radices[i];
        p.mq       = magic(ns);
        p.mg       = magic(p.nbf);
        p.fast     = layout == RP_COLS || (layout == RP_ROWS && i > 0);
        p.tw_off   = off;
        if (ns > 1)
            off += ns * (radices[i] - 1);
        p.wr_off = off;
        if (radices[i] > kRpMaxRadix)
            off += radices[i];
        ns *= radices[i];
    }
    const bool fl = layout != RP_SIGNALS;
    for (int i = 0; i + 1 < d.npass; i++)
    {
        const int nn  = d.pass[i].ns * d.pass[i].radix;
        const int tot = fl ? S : 4;
        int best = 0, best_c = -1;
        for (int pad : { 0, 1, 2, 3, 4, 6, 8 })
        {
            if (pad * 4 > nn * (fl ? S : 1))
                break;
            set_layout(d, i, S, fl, pad);
            const int ta = tot * d.pass[i].nbf, tb = tot * d.pass[i + 1].nbf;
            int c = 0;
            for (int w = 0; w < 3 && (best_c < 0 || c < best_c); w++)
            {
                const int fa = w * (ta / 3) / 32 * 32, fb = w * (tb / 3) / 32 * 32;
                c += d.pass[i].radix * store_conflicts(d.pass[i], d.shift, elem, fa, ta);
                c += d.pass[i + 1].radix * load_conflicts(d.pass[i + 1], d.shift, elem, fb, tb);
            }
            if (best_c < 0 || c < best_c)
            {
                best_c = c;
                best   = pad;
            }
            if (c == 0)
                break;
        }
        set_layout(d, i, S, fl, best);
    }
    if (d.npass > 0)
    {
        // the natural layout of a single pass, or of the ends of a transform from and to shared memory
        rp_pass& f = d.pass[0];
        rp_pass& l = d.pass[d.npass - 1];
        if (smem_io || d.npass == 1)
        {
            const int e = fl ? S : 1, sg = fl ? 1 : d.n;
            f.ld_e = e;
            f.ld_q = 0;
            f.ld_g = sg;
            f.ld_r = f.nbf * e;
            l.st_e = e;
            l.st_q = d.n * e;
            l.st_g = sg;
            l.st_r = l.ns * e;
        }
    }
    d.elems = rp_smem_elems(d, layout, S, smem_io);
    return d;
}

int rp_smem_elems(const rp_desc& d, rp_layout layout, int S, bool smem_io)
{
    int m = smem_io || d.npass == 1 ? (layout == RP_SIGNALS ? d.n : d.n * S) : 0;
    for (int i = 0; i + 1 < d.npass; i++)
    {
        const rp_pass& p = d.pass[i];
        const int groups = d.n / (p.ns * p.radix);
        m                = std::max(m, groups * p.st_q);
    }
    return m;
}

int rp_threads_needed(const rp_desc& d, int nsig, bool smem_io)
{
    int t = 1;
    for (int i = smem_io ? 0 : 1; i < d.npass - (smem_io ? 0 : 1); i++)
    {
        const int R = d.pass[i].radix;
        const int h = R > kRpMaxRadix ? d.hold : rp_held(R, d.hold);
        t = std::max(t, ((R > kRpMaxRadix ? nsig * d.n : nsig * d.pass[i].nbf) + h - 1) / h);
    }
    return t;
}

static double efficiency(const rp_desc& d, int spc, int threads)
{
    double useful = 0, spent = 0;
    for (int i = 0; i < d.npass; i++)
    {
        const rp_pass& p = d.pass[i];
        const double w   = rp_pass_cost(p.radix) * p.radix;
        const int bf     = spc * p.nbf;
        useful += w * bf;
        spent += w * double((bf + threads - 1) / threads) * threads;
    }
    return useful / spent;
}

bool rp_fits(const std::vector<int>& radices, int elem, int smem_budget, bool smem_io, int hold)
{
    long long n = 1, widest = 1;
    for (int r : radices)
        n *= r;
    for (size_t i = smem_io ? 0 : 1; i < radices.size() && (smem_io || i + 1 < radices.size()); i++)
    {
        const int R = radices[i];
        const int h = R > kRpMaxRadix ? hold : rp_held(R, hold);
        widest      = std::max(widest, ((R > kRpMaxRadix ? n : n / R) + h - 1) / h);
    }
    return !radices.empty() && widest <= rp_max_threads(elem, hold) && n * elem / 16 * 17 + 64 <= smem_budget;
}

rp_shape rp_choose(const rp_desc& d, int sig_elems, int elem, int smem_budget, bool smem_io)
{
    // the most busy threads per SM: how evenly the passes' butterflies fill the threads times how many
    // threads are resident (64 registers each), small CTAs first so that one CTA's barriers and global
    // accesses overlap with others' work
    rp_shape best;
    double score   = 0;
    const int maxt = rp_max_threads(elem, d.hold);
    int most = 1; // butterflies (dot products of a prime radix) of a signal's largest pass
    for (int i = 0; i < d.npass; i++)
        most = std::max(most, d.pass[i].radix > kRpMaxRadix ? d.n : d.pass[i].nbf);
    for (int threads : { 64, 96, 128, 160, 192, 224, 256, 320, 384, 448, 512, 640, 768, 896, 1024 })
        for (int spc = std::max(1, threads / (2 * most)), tried = 0; threads <= maxt && tried < 24; spc++, tried++)
        {
            if (rp_threads_needed(d, spc, smem_io) > threads)
                break;
            const long long smem = (long long)spc * sig_elems * elem;
            if (smem > smem_budget || (spc > 1 && (long long)spc * d.n > 8LL * threads * 16 / 8))
                break;
            const int ctas     = std::min({ int((smem_budget + 1024) / (smem + 2048)), maxt / threads, 24 });
            const int resident = std::max(1, ctas) * threads;
            double s           = efficiency(d, spc, threads) * std::min(1.0, resident / (0.94 * maxt));
            if (ctas < 3)
                s *= ctas < 2 ? 0.75 : 0.92;
            if (threads > 256)
                s *= 0.97;
            if (s > score * 1.01)
            {
                score = s;
                best  = { spc, threads };
            }
        }
    return best;
}

rp_shape rp_shrink(const rp_desc& d, const rp_shape& full, long long batch, int sms, bool smem_io)
{
    if (batch >= 2LL * sms * full.spc)
        return full;
    rp_shape s;
    s.spc  = int(std::min<long long>(full.spc, (batch + 2LL * sms - 1) / (2LL * sms))); // at most two CTAs per SM
    int bf = 1;
    for (int i = 0; i < d.npass; i++)
        bf = std::max(bf, s.spc * (d.pass[i].radix > kRpMaxRadix ? d.n : d.pass[i].nbf));
    const int need = rp_threads_needed(d, s.spc, smem_io);
    s.threads      = (std::max(need, std::min(bf, d.hold == kRpHold ? 512 : 256)) + 31) / 32 * 32;
    return s;
}

int rp_tile(const std::vector<int>& radices, int elem, int smem_budget, int hold)
{
    long long n = 1;
    for (int r : radices)
        n *= r;
    int widest = 1; // butterflies per column the in-place passes hold at once, threads each
    for (size_t i = 1; i + 1 < radices.size(); i++)
    {
        const int R = radices[i];
        const int h = R > kRpMaxRadix ? hold : rp_held(R, hold);
        widest      = std::max<long long>(widest, ((R > kRpMaxRadix ? n : n / R) + h - 1) / h);
    }
    int S = 128 / elem;
    while (n * S < 512)
        S *= 2;
    // 64-byte rows while that gives four CTAs per SM instead of two, four columns for two CTAs instead of one (complex
    // float: eight 1080 x 1920 arrays 174 -> 155 us with 4 columns instead of 8, sixteen 512 x 512 35 -> 33 us with 8
    // instead of 16, 32 signals of 250000 points 108 -> 96 us; complex double is bound by its arithmetic, +-2%)
    while (S * elem > 64 && S * widest > rp_max_threads(elem, hold) / 4)
        S /= 2;
    while (S > 4 && S * widest > rp_max_threads(elem, hold) / 2)
        S /= 2;
    for (; S >= 1; S /= 2)
        if ((long long)S * widest <= rp_max_threads(elem, hold) && n * S * elem / 16 * 17 <= smem_budget)
            return S;
    return 0;
}

} // namespace kfr_gpu
