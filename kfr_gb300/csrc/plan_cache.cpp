// Plans kept between calls (see convolve.hpp).  Their tables are device memory, so a plan belongs to the device that was
// current when it was built.
#include "conv.hpp"
#include "convolve.hpp"
#include "workspace.hpp"

namespace kfr_gpu
{

struct plan_cache::entry
{
    int kind, device;
    long long n;
    std::shared_ptr<void> plan;
};

plan_cache& plan_cache::instance()
{
    static plan_cache c;
    return c;
}

template <class P, class BUILD>
std::shared_ptr<P> plan_cache::get(int kind, long long n, const BUILD& build)
{
    int device = 0;
    check(cudaGetDevice(&device), "current device");
    std::lock_guard<std::mutex> lock(mu_);
    for (auto& e : entries_)
        if (e->kind == kind && e->device == device && e->n == n)
            return std::static_pointer_cast<P>(e->plan);
    std::shared_ptr<P> p = build();
    entries_.push_back(std::make_shared<entry>(entry{ kind, device, n, p }));
    return p;
}

template <typename T>
std::shared_ptr<complex_engine<T>> plan_cache::complex(long long n)
{
    return get<complex_engine<T>>(sizeof(T) == 8, n, [&]() { return std::make_shared<complex_engine<T>>(n); });
}

template <typename T>
std::shared_ptr<real_engine<T>> plan_cache::real(long long n)
{
    return get<real_engine<T>>(2 + (sizeof(T) == 8), n, [&]() { return std::make_shared<real_engine<T>>(n); });
}

template <typename T>
std::shared_ptr<fir_tables<T>> plan_cache::fir(long long n, bool paired)
{
    return get<fir_tables<T>>(4 + (sizeof(T) == 8) + (paired ? 2 : 0), n,
                              [&]()
                              {
                                  auto p = std::make_shared<fir_tables<T>>(size_t(n), paired);
                                  p->roots64(size_t(n));
                                  return p;
                              });
}

void plan_cache::clear()
{
    std::lock_guard<std::mutex> lock(mu_);
    entries_.clear();
    workspace_trim();
}

size_t plan_cache::size() const
{
    std::lock_guard<std::mutex> lock(mu_);
    return entries_.size();
}

template std::shared_ptr<complex_engine<float>> plan_cache::complex<float>(long long);
template std::shared_ptr<complex_engine<double>> plan_cache::complex<double>(long long);
template std::shared_ptr<real_engine<float>> plan_cache::real<float>(long long);
template std::shared_ptr<real_engine<double>> plan_cache::real<double>(long long);
template std::shared_ptr<fir_tables<float>> plan_cache::fir<float>(long long, bool);
template std::shared_ptr<fir_tables<double>> plan_cache::fir<double>(long long, bool);

} // namespace kfr_gpu
