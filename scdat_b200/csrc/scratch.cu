// scratch.cu -- the scratch pools (see scratch.cuh).
#include "scratch.cuh"

#include <mutex>

namespace scdat {

namespace {

constexpr int kMaxDevices = 64;
std::mutex g_mu;
cudaMemPool_t g_pool[kMaxDevices] = {};

cudaError_t pool_of_device(cudaMemPool_t* pool)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(g_mu);
    if (!g_pool[dev]) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.handleTypes = cudaMemHandleTypeNone;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t q = nullptr;
        e = cudaMemPoolCreate(&q, &props);
        if (e != cudaSuccess) return e;
        unsigned long long keep = kScratchKeep;
        e = cudaMemPoolSetAttribute(q, cudaMemPoolAttrReleaseThreshold, &keep);
        if (e != cudaSuccess) {
            cudaMemPoolDestroy(q);
            return e;
        }
        g_pool[dev] = q;
    }
    *pool = g_pool[dev];
    return cudaSuccess;
}

thread_local SpareScope* t_spare = nullptr;

}  // namespace

SpareScope::SpareScope(bool (*give_back)(void*), void* who) : give_back_(give_back), who_(who), outer_(t_spare)
{
    t_spare = this;
}

SpareScope::~SpareScope() { t_spare = outer_; }

bool spare_give_back()
{
    SpareScope* s = t_spare;
    if (!s || !s->give_back_) return false;
    SpareScope none(nullptr, nullptr);  // what give_back allocates itself has nothing to fall back on
    return s->give_back_(s->who_);
}

cudaError_t scratch_alloc(void** p, size_t bytes, cudaStream_t st)
{
    cudaMemPool_t pool = nullptr;
    cudaError_t e = pool_of_device(&pool);
    if (e != cudaSuccess) return e;
    e = cudaMallocFromPoolAsync(p, bytes, pool, st);
    while (e == cudaErrorMemoryAllocation && spare_give_back()) {
        cudaGetLastError();
        e = cudaMallocFromPoolAsync(p, bytes, pool, st);
    }
    return e;
}

void scratch_free(void* p, cudaStream_t st) { cudaFreeAsync(p, st); }

void scratch_trim()
{
    std::lock_guard<std::mutex> lock(g_mu);
    for (cudaMemPool_t q : g_pool)
        if (q) cudaMemPoolTrimTo(q, 0);
}

}  // namespace scdat
