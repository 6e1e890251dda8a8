// Builds plans on the CPU (cuda_stub.cpp).
//   test_plan_lengths f|d LO HI    complex, real and DCT plans of every length of LO .. HI with a one-CTA transform,
//                                 in single or double precision; the in-place passes held by their threads, their
//                                 addresses inside the tile
//   test_plan_lengths sf|sd N...  the strategy of the complex plans
//   test_plan_lengths rf|rd N...  the launches of the real plans' forward transforms and their descriptions
#include "plan.hpp"

#include <cstdio>
#include <cstdlib>

using namespace kfr_gpu;

template <class F>
static bool builds(const char* what, long long n, const F& f)
{
    try
    {
        f();
        return true;
    }
    catch (const std::exception& e)
    {
        std::printf("%s of %lld: %s\n", what, n, e.what());
        return false;
    }
}

#define CHECK(c)                                                                                           \
    do                                                                                                     \
    {                                                                                                      \
        if (!(c))                                                                                          \
        {                                                                                                  \
            std::printf("in-place transform of %d: %s\n", p.n, #c);                                        \
            return false;                                                                                  \
        }                                                                                                  \
    } while (0)

template <typename T>
static bool in_place(const block_program<T>& p)
{
    if (p.ct)
        return true;
    const rp_desc& d = p.desc;
    for (long long batch : { 1LL, 9LL, 100000LL })
    {
        const block_cfg c = p.cfg(batch);
        CHECK(c.spc >= 1 && c.grid * c.spc >= batch && c.smem == c.spc * d.elems * int(2 * sizeof(T)));
        CHECK(c.smem <= smem_budget() && c.threads <= rp_max_threads(2 * sizeof(T), d.hold));
        CHECK(rp_threads_needed(d, c.spc, true) <= c.threads);
    }
    int n = 1;
    for (int i = 0; i < d.npass; i++)
    {
        const rp_pass& q = d.pass[i];
        CHECK(q.ns == n && q.nbf * q.radix == d.n);
        n *= q.radix;
        for (int j = 0; j < q.nbf; j++)
        {
            const int a = j / q.ns, k = j % q.ns, r = q.radix - 1;
            CHECK(j * q.ld_e + a * q.ld_q + r * q.ld_r < d.elems && k * q.st_e + a * q.st_q + r * q.st_r < d.elems);
        }
    }
    CHECK(n == d.n);
    return true;
}

template <typename T>
static bool check(long long lo, long long hi)
{
    bool ok = true;
    for (long long n = lo; n <= hi; n++)
    {
        if (!rp_program<T>::feasible(n))
            continue;
        ok &= builds("complex DFT", n, [&]() { complex_engine<T> e(n); });
        ok &= builds("real DFT", 2 * n, [&]() { real_engine<T> e(2 * n); });
        ok &= builds("DCT", n, [&]() { dct_engine<T> e(n); });
        block_program<T> p;
        ok &= builds("in-place transform", n, [&]() { p.build(int(n), CT_REAL); }) && in_place(p);
    }
    return ok;
}

template <typename T>
static void strategies(int argc, char** argv)
{
    using kind = typename complex_engine<T>::kind;
    for (int i = 2; i < argc; i++)
    {
        const kind k = complex_engine<T>(std::atoll(argv[i])).strategy();
        std::printf("%s ", k == kind::smem              ? "direct"
                           : k == kind::fourstep        ? "fourstep"
                           : k == kind::rader_smem      ? "rader"
                           : k == kind::bluestein_smem  ? "bluestein"
                           : k == kind::bluestein_multi ? "multi"
                                                        : "other");
    }
}

template <typename T>
static void reals(int argc, char** argv)
{
    for (int i = 2; i < argc; i++)
    {
        const real_engine<T> e(std::atoll(argv[i]));
        std::printf("%d %s\n", e.launches(3), e.describe().c_str());
    }
}

int main(int argc, char** argv)
{
    if (argv[1][0] == 'r')
    {
        argv[1][1] == 'f' ? reals<float>(argc, argv) : reals<double>(argc, argv);
        return 0;
    }
    if (argv[1][0] == 's')
    {
        argv[1][1] == 'f' ? strategies<float>(argc, argv) : strategies<double>(argc, argv);
        return 0;
    }
    const long long lo = std::atoll(argv[2]), hi = std::atoll(argv[3]);
    const bool ok = argv[1][0] == 'f' ? check<float>(lo, hi) : check<double>(lo, hi);
    std::printf("%s\n", ok ? "ok" : "failed");
    return !ok;
}
