// Linked with the library's objects and --wrap into a second library whose cooperative launches and
// device allocations a test can make fail on the host.
#include <cuda_runtime.h>

#include <map>
#include <mutex>

extern "C" {
cudaError_t __real_cudaLaunchCooperativeKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t);
cudaError_t __real_cudaMalloc(void**, size_t);
cudaError_t __real_cudaFree(void*);
cudaError_t __real_cudaMemGetInfo(size_t*, size_t*);

static int g_refuse = 0, g_short = 0, g_calls = 0;
static size_t g_budget = 0, g_used = 0;
static std::map<void*, size_t> g_size;
static std::mutex g_mu;

// refuse: every cooperative launch is too large.  short_launch: the n-th from now on leaves out its last
// block, so that the waits for it run out (0: none).
__attribute__((visibility("default"))) void fault_launches(int refuse, int short_launch)
{
    g_refuse = refuse;
    g_short = short_launch;
    g_calls = 0;
}
__attribute__((visibility("default"))) int fault_calls() { return g_calls; }

// the device has this many bytes (0: what it has)
__attribute__((visibility("default"))) void fault_budget(size_t bytes) { g_budget = bytes; }
__attribute__((visibility("default"))) size_t fault_used() { return g_used; }

cudaError_t __wrap_cudaLaunchCooperativeKernel(const void* f, dim3 grid, dim3 block, void** args, size_t smem,
                                               cudaStream_t st)
{
    ++g_calls;
    if (g_refuse) return cudaErrorCooperativeLaunchTooLarge;
    if (g_short == g_calls) --grid.x;
    return __real_cudaLaunchCooperativeKernel(f, grid, block, args, smem, st);
}

cudaError_t __wrap_cudaMalloc(void** p, size_t bytes)
{
    std::lock_guard<std::mutex> lock(g_mu);
    if (g_budget && g_used + bytes > g_budget) return cudaErrorMemoryAllocation;
    const cudaError_t e = __real_cudaMalloc(p, bytes);
    if (e == cudaSuccess) g_used += g_size[*p] = bytes;
    return e;
}

cudaError_t __wrap_cudaFree(void* p)
{
    std::lock_guard<std::mutex> lock(g_mu);
    const auto it = g_size.find(p);
    if (it != g_size.end()) {
        g_used -= it->second;
        g_size.erase(it);
    }
    return __real_cudaFree(p);
}

cudaError_t __wrap_cudaMemGetInfo(size_t* free, size_t* total)
{
    const cudaError_t e = __real_cudaMemGetInfo(free, total);
    if (e == cudaSuccess && g_budget) {
        *total = g_budget;
        *free = g_budget > g_used ? g_budget - g_used : 0;
    }
    return e;
}
}
