// Builds plans on the CPU (cuda_stub.cpp).
//   test_plan_lengths f|d LO HI    complex, real and DCT plans of every length of LO .. HI with a one-CTA transform,
//                                 in single or double precision
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
    }
    return ok;
}

int main(int, char** argv)
{
    const long long lo = std::atoll(argv[2]), hi = std::atoll(argv[3]);
    const bool ok = argv[1][0] == 'f' ? check<float>(lo, hi) : check<double>(lo, hi);
    std::printf("%s\n", ok ? "ok" : "failed");
    return !ok;
}
