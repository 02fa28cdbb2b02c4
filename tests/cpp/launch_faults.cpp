// Linked with the library's objects and --wrap into a second library whose cooperative launches and
// device allocations a test can make fail on the host.
#include <cuda_runtime.h>

extern "C" {
cudaError_t __real_cudaLaunchCooperativeKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t);
cudaError_t __real_cudaMalloc(void**, size_t);

static int g_refuse = 0, g_short = 0, g_calls = 0;
static size_t g_limit = 0;

// refuse: every cooperative launch is too large.  short_launch: the n-th from now on leaves out its last
// block, so that the waits for it run out (0: none).
__attribute__((visibility("default"))) void fault_launches(int refuse, int short_launch)
{
    g_refuse = refuse;
    g_short = short_launch;
    g_calls = 0;
}
__attribute__((visibility("default"))) int fault_calls() { return g_calls; }

// allocations above this many bytes fail (0: none do)
__attribute__((visibility("default"))) void fault_alloc_above(size_t bytes) { g_limit = bytes; }

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
    if (g_limit && bytes > g_limit) return cudaErrorMemoryAllocation;
    return __real_cudaMalloc(p, bytes);
}
}
