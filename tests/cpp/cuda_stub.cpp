// The CUDA calls and kernel queries that building a plan makes, for tests without a GPU: device memory is host memory,
// no kernel has a compile-time variant of its own, and kernels are never launched (link with unresolved symbols
// allowed).
#include <cstdlib>
#include <cstring>
#include <vector>
#include <cuda_runtime.h>

int g_stub_device = 0; // the current device

extern "C"
{
cudaError_t cudaMalloc(void** p, size_t n)
{
    *p = std::malloc(n ? n : 1);
    return cudaSuccess;
}
cudaError_t cudaFree(void* p)
{
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind)
{
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n)
{
    std::memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned)
{
    *p = std::malloc(n);
    return cudaSuccess;
}
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned)
{
    *d = h;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d)
{
    *d = g_stub_device;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "stub"; }
}

namespace kfr_gpu
{
int max_smem_bytes() { return 227 * 1024; }
bool ct_square_f32(long long, std::vector<int>&) { return false; }
bool has_ct_fsp_r2c_f32(int, int) { return false; }
bool rader_pfa_shape(long long, std::vector<int>&, int&) { return false; }
void workspace_trim() {}
} // namespace kfr_gpu
