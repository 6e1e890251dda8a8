// Stream-ordered workspaces of calls that need device memory only while they run.
//
// They come from a memory pool of this library's own (one per device), which keeps up to kWorkspaceKeep bytes
// between calls (cudaMallocAsync's default pool returns everything at each synchronisation and maps it again
// on the next call) and gives them back when the plan cache is cleared.  Safe from several threads and
// streams: allocations and frees are ordered by the stream they are made on.
#pragma once

#include <cstddef>
#include <cuda_runtime.h>

namespace kfr_gpu
{

constexpr size_t kWorkspaceKeep = size_t(64) << 20;

class workspace
{
public:
    workspace(size_t bytes, cudaStream_t st);
    ~workspace();
    workspace(const workspace&)            = delete;
    workspace& operator=(const workspace&) = delete;
    void* get() const { return p_; }

private:
    void* p_ = nullptr;
    cudaStream_t st_;
};

// Returns the memory the pools keep.
void workspace_trim();

} // namespace kfr_gpu
