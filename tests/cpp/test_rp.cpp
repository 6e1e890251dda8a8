// Walks the descriptors of rp.hpp on the CPU: every shared-memory address in range and written once per pass,
// every middle butterfly held by a thread, and the transform of random signals equal to the direct DFT.
//   test_rp LAYOUT S ELEM SMEM_IO HOLD N...      (LAYOUT 0 signals, 1 columns, 2 rows)
#include "rp.hpp"

#include <cmath>
#include <complex>
#include <cstdio>
#include <cstdlib>
#include <random>

using namespace kfr_gpu;
using cd = std::complex<double>;

static cd root(long long k, long long n)
{
    const double a = -2.0 * M_PI * double(k % n) / double(n);
    return { std::cos(a), std::sin(a) };
}
static int mulhi(int a, uint32_t m) { return int((uint64_t(uint32_t(a)) * m) >> 32); }

#define CHECK(c)                                                                                           \
    do                                                                                                     \
    {                                                                                                      \
        if (!(c))                                                                                          \
        {                                                                                                  \
            std::printf("n=%d pass %d: %s\n", d.n, i, #c);                                                \
            return false;                                                                                  \
        }                                                                                                  \
    } while (0);

static bool run(int n, rp_layout layout, int S, int elem, bool io, int hold)
{
    const auto rad = rp_radices(n, 127, hold);
    if (rad.empty())
        return false;
    for (int r : rad)
        if (r > kRpMaxRadix)
            for (int q = 2; q < r; q++)
                if (r % q == 0)
                {
                    std::printf("n=%d: composite radix %d without a codelet\n", n, r);
                    return false;
                }
    const rp_desc d = rp_build(rad, layout, S, elem, io, hold);
    const int nsig  = layout == RP_SIGNALS ? (n > 512 ? 2 : 5) : S;
    const int elems = rp_smem_elems(d, layout, S, io) * (layout == RP_SIGNALS ? nsig : 1);
    const int thr   = rp_threads_needed(d, nsig, io);
    std::mt19937 gen(n);
    std::uniform_real_distribution<double> u(-1, 1);
    std::vector<std::vector<cd>> x(nsig, std::vector<cd>(n)), y(nsig, std::vector<cd>(n));
    for (auto& v : x)
        for (auto& e : v)
            e = { u(gen), u(gen) };
    std::vector<cd> buf(elems);
    int i = 0;
    if (io)
        for (int g = 0; g < nsig; g++)
            for (int e = 0; e < n; e++)
                buf[g * n + e] = x[g][e];
    for (i = 0; i < d.npass; i++)
    {
        const rp_pass& p = d.pass[i];
        const bool first = i == 0 && !io, last = i == d.npass - 1 && !io;
        const int total  = nsig * p.nbf;
        if (!first && !last)
        {
            if (p.radix > kRpMaxRadix)
                { CHECK((total * p.radix + hold - 1) / hold <= thr) }
            else
                { CHECK((total + rp_held(p.radix, hold) - 1) / rp_held(p.radix, hold) <= thr) }
        }
        else
            { CHECK(p.radix <= kRpMaxRadix) }
        std::vector<cd> next(elems);
        std::vector<char> seen(elems), read(elems);
        for (int J = 0; J < total; J++)
        {
            int g, j;
            if (p.fast)
                g = J & ((1 << d.shift) - 1), j = J >> d.shift;
            else
                g = p.mg ? mulhi(J, p.mg) : J, j = J - g * p.nbf;
            CHECK(g >= 0 && g < nsig && j >= 0 && j < p.nbf)
            const int q = p.mq ? mulhi(j, p.mq) : j, k = j - q * p.ns;
            CHECK(q == j / p.ns && k == j % p.ns)
            std::vector<cd> v(p.radix), o(p.radix);
            for (int r = 0; r < p.radix; r++)
            {
                const int a = j * p.ld_e + q * p.ld_q + g * p.ld_g + r * p.ld_r;
                if (!first)
                {
                    CHECK(a >= 0 && a < elems)
                    CHECK(!read[a])
                    read[a] = 1;
                }
                v[r] = (first ? x[g][j + r * p.nbf] : buf[a]) * root((long long)k * r, (long long)p.ns * p.radix);
            }
            for (int s = 0; s < p.radix; s++)
                for (int r = 0; r < p.radix; r++)
                    o[s] += v[r] * root((long long)s * r, p.radix);
            for (int r = 0; r < p.radix; r++)
            {
                const int a = k * p.st_e + q * p.st_q + g * p.st_g + r * p.st_r;
                if (last && d.npass > 1)
                {
                    y[g][k + r * p.ns] = o[r];
                    continue;
                }
                CHECK(a >= 0 && a < elems)
                CHECK(!seen[a])
                seen[a] = 1;
                next[a] = o[r];
            }
        }
        buf = next;
    }
    if (io || d.npass == 1)
        for (int g = 0; g < nsig; g++)
            for (int e = 0; e < n; e++)
                y[g][e] = io ? buf[layout == RP_SIGNALS ? g * n + e : e * S + g]
                             : buf[e * d.pass[0].st_r + g * d.pass[0].st_g];
    double err = 0, ref = 0;
    for (int g = 0; g < nsig; g++)
        for (int k = 0; k < n; k += (n > 600 ? n / 97 + 1 : 1))
        {
            cd s = 0;
            for (int e = 0; e < n; e++)
                s += x[g][e] * root((long long)k * e, n);
            err += std::norm(s - y[g][k]);
            ref += std::norm(s);
        }
    if (!(err <= 1e-22 * ref))
    {
        std::printf("n=%d: error %g\n", n, std::sqrt(err / ref));
        return false;
    }
    // launch shapes: every in-place butterfly has a thread, the tile fits
    const int sig = rp_smem_elems(d, RP_SIGNALS, 1, io);
    if (layout == RP_SIGNALS)
    {
        const rp_shape s = rp_choose(d, sig, elem, 220 * 1024, io);
        for (long long batch : { 1LL, 7LL, 300LL, 5000LL, 1000000LL })
        {
            const rp_shape t = rp_shrink(d, s, batch, 152, io);
            if (s.spc && !(t.spc >= 1 && t.spc <= s.spc && t.threads % 32 == 0 && t.threads <= rp_max_threads(elem, hold) &&
                           rp_threads_needed(d, t.spc, io) <= t.threads && (long long)t.spc * sig * elem <= 220 * 1024))
            {
                std::printf("n=%d batch %lld: shape %d x %d\n", n, batch, t.spc, t.threads);
                return false;
            }
        }
        if (std::getenv("RP_SHOW"))
        {
            std::printf("n=%d spc=%d threads=%d elems=%d radices", n, s.spc, s.threads, sig);
            for (int r : rad)
                std::printf(" %d", r);
            std::printf("\n");
        }
    }
    return true;
}

int main(int argc, char** argv)
{
    const auto layout = rp_layout(std::atoi(argv[1]));
    const int S = std::atoi(argv[2]), elem = std::atoi(argv[3]), io = std::atoi(argv[4]),
              hold = std::atoi(argv[5]);
    for (int i = 6; i < argc; i++)
        if (!run(std::atoi(argv[i]), layout, S, elem, io != 0, hold))
            return 1;
    std::printf("ok\n");
    return 0;
}
