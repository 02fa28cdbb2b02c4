// scratch.cuh -- stream-ordered scratch memory for calls that need buffers only while they run
// (scdat_pcg_csr, the adjoint window).  It comes from a memory pool of this library's own, one per
// device, that keeps up to kScratchKeep bytes between calls: a cudaMalloc and cudaFree per buffer
// took longer than the work (a CSR solve of 110k rows 1.0 ms of 4.1, an adjoint window of 16^3 cells
// 5.5 of 19.9).  What lies above that goes back to the device at the next synchronisation, and all
// of it when an allocation of this library fails.  The runtime's pools are safe to use from several
// threads, and a buffer is reused on another stream only once the stream that freed it has got there.
#pragma once

#include <cstddef>
#include <cuda_runtime.h>

namespace scdat {

constexpr size_t kScratchKeep = 128ull << 20;

cudaError_t scratch_alloc(void** p, size_t bytes, cudaStream_t st);
void scratch_free(void* p, cudaStream_t st);
void scratch_trim();  // gives the kept memory of every device back

// Memory a call on this thread can do without, given back when an allocation fails: give_back frees some
// and returns true, or returns false.  Scopes nest; one of a null function has none to give.
class SpareScope {
public:
    SpareScope(bool (*give_back)(void*), void* who);
    ~SpareScope();
    SpareScope(const SpareScope&) = delete;
    SpareScope& operator=(const SpareScope&) = delete;

private:
    bool (*give_back_)(void*);
    void* who_;
    SpareScope* outer_;
    friend bool spare_give_back();
};
bool spare_give_back();

// A scratch buffer of n values on one stream.
template <typename T>
struct SBuf {
    T* p = nullptr;
    size_t n = 0;
    cudaStream_t st = nullptr;
    SBuf() = default;
    SBuf(const SBuf&) = delete;
    SBuf& operator=(const SBuf&) = delete;
    ~SBuf() { release(); }
    void release()
    {
        if (p) scratch_free(p, st);
        p = nullptr;
        n = 0;
    }
    cudaError_t alloc(size_t count, cudaStream_t on)
    {
        release();
        st = on;
        if (count == 0) return cudaSuccess;
        const cudaError_t e = scratch_alloc((void**)&p, count * sizeof(T), on);
        if (e == cudaSuccess) n = count;
        return e;
    }
};

}  // namespace scdat
