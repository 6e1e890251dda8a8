// Stream-ordered workspaces (see workspace.hpp).
#include "workspace.hpp"
#include "plan.hpp"

#include <map>
#include <mutex>

namespace kfr_gpu
{

namespace
{
std::mutex g_mu;
std::map<int, cudaMemPool_t> g_pools;

cudaMemPool_t pool_of_device()
{
    int dev = 0;
    check(cudaGetDevice(&dev), "current device");
    std::lock_guard<std::mutex> lock(g_mu);
    auto f = g_pools.find(dev);
    if (f != g_pools.end())
        return f->second;
    cudaMemPoolProps props{};
    props.allocType     = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id   = dev;
    cudaMemPool_t pool  = nullptr;
    check(cudaMemPoolCreate(&pool, &props), "create workspace pool");
    unsigned long long keep = kWorkspaceKeep;
    check(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep), "workspace pool threshold");
    g_pools[dev] = pool;
    return pool;
}
} // namespace

workspace::workspace(size_t bytes, cudaStream_t st) : st_(st)
{
    if (bytes)
        check(cudaMallocFromPoolAsync(&p_, bytes, pool_of_device(), st), "allocate workspace");
}

workspace::~workspace()
{
    if (p_)
        cudaFreeAsync(p_, st_);
}

void workspace_trim()
{
    std::lock_guard<std::mutex> lock(g_mu);
    for (auto& p : g_pools)
        cudaMemPoolTrimTo(p.second, 0);
}

} // namespace kfr_gpu
