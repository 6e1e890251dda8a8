// The plan cache on the CPU (cuda_stub.cpp): one plan per precision, kind, length and device.
#include "convolve.hpp"

#include <cstdio>

using namespace kfr_gpu;

extern int g_stub_device;

#define CHECK(c)                                                                                           \
    do                                                                                                     \
    {                                                                                                      \
        if (!(c))                                                                                          \
        {                                                                                                  \
            std::printf("line %d: %s\n", __LINE__, #c);                                                   \
            return 1;                                                                                      \
        }                                                                                                  \
    } while (0)

int main()
{
    plan_cache& c = plan_cache::instance();
    g_stub_device = 0;
    const auto a  = c.complex<float>(360);
    const auto r  = c.real<float>(360);
    g_stub_device = 1;
    const auto b  = c.complex<float>(360);
    CHECK(a != b && c.size() == 3);
    CHECK(c.real<float>(360) != r && c.size() == 4);
    CHECK(c.complex<float>(360) == b && c.size() == 4);
    g_stub_device = 0;
    CHECK(c.complex<float>(360) == a && c.real<float>(360) == r && c.size() == 4);
    c.clear();
    CHECK(c.size() == 0);
    std::printf("ok\n");
    return 0;
}
