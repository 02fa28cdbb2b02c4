// pcg_group.cu -- launches of the one-launch Jacobi-PCG (pcg_group.cuh) on a single system.
#include "pcg_group.cuh"

#include <algorithm>

namespace scdat {

namespace {

template <int J, int K>
__global__ void __launch_bounds__(kCgMaxThreads, 1)
    k_cg64(const __grid_constant__ PoissonView A, const double* b, double* x, double2* zp, PcgScalars* sc,
           unsigned long long* slots, unsigned vgrid, double rtol, int max_iter, int smem_bytes)
{
    extern __shared__ __align__(16) unsigned char smem[];
    CgGroup g{blockIdx.x, gridDim.x, slots, vgrid};
    cg_solve64<J, K>(g, A, b, x, zp, sc, rtol, max_iter, smem, smem_bytes);
}

template <int J, int K>
__global__ void __launch_bounds__(kCgMaxThreads, 1)
    k_cg_mixed(const __grid_constant__ PoissonView A, const double* b, double* x, double2* zp, PcgScalars* sc,
               unsigned long long* slots, unsigned vgrid, double rtol, int max_iter, int smem_bytes)
{
    extern __shared__ __align__(16) unsigned char smem[];
    CgGroup g{blockIdx.x, gridDim.x, slots, vgrid};
    cg_solve_mixed<J, K>(g, A, b, x, zp, sc, rtol, max_iter, smem, smem_bytes);
}

template <typename K>
cudaError_t launch_group(K kernel, const CgPlan& plan, void** args, cudaStream_t st)
{
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kCgSmemBytes);
    if (e != cudaSuccess) return e;
    return cg_launch((const void*)kernel, plan.blocks, plan.threads, args, (size_t)plan.smem, st);
}

}  // namespace

CgPlan cg_plan(const int* rows, const int* grids, int n, int nsm, int* blocks_of)
{
    CgPlan plan;
    if (nsm > kCgMaxGroup) nsm = kCgMaxGroup;
    int most = 0, rounds = 1;
    for (int k = 0; k < n; ++k) {
        const int64_t span = (int64_t)grids[k] * kCgVirtual;
        most = std::max(most, rows[k]);
        rounds = (int)std::max<int64_t>(rounds, (rows[k] + span - 1) / span);
    }
    const bool one_block = most > kCgVirtual && most <= kCgMaxThreads;
    for (int j = 1; j * (int64_t)rounds <= kCgRowsPerThread; ++j)
        for (int threads = j * rounds == 1 && !one_block ? kCgVirtual : kCgMaxThreads; threads <= kCgMaxThreads;
             threads *= 2) {
            int64_t blocks = 0;
            for (int k = 0; k < n; ++k) {
                const int per = j * threads / kCgVirtual;  // virtual blocks of a block
                const int virt = std::min(grids[k], (rows[k] + kCgVirtual - 1) / kCgVirtual);
                blocks_of[k] = std::max(1, (virt + per - 1) / per);
                blocks += blocks_of[k];
            }
            if (blocks > nsm) continue;
            plan.threads = threads;
            plan.virt = j;
            plan.rounds = rounds;
            plan.rows_per_thread = j * rounds;
            plan.blocks = (int)blocks;
            const int64_t want = (int64_t)threads * j * rounds * kCgRowSlots * kCgEntryBytes;
            plan.smem = (int)(want < kCgSmemBytes ? want : kCgSmemBytes);
            plan.planes = j * threads / kCgVirtual > 4 ? 2 : 1;  // two dots of each virtual block
            plan.ok = true;
            return plan;
        }
    return plan;
}

cudaError_t launch_cg64(const CgPlan& plan, int grid, const PoissonView& A, const double* b, double* x, double* zp,
                        PcgScalars* sc, double* slots, double rtol, int max_iter, cudaStream_t st)
{
    cudaError_t e = cudaMemsetAsync(slots, 0, plan.planes * kCgPlaneBytes, st);
    if (e != cudaSuccess) return e;
    int smem = plan.smem;
    void* args[] = {(void*)&A, &b, &x, &zp, &sc, &slots, &grid, &rtol, &max_iter, &smem};
    return cg_dispatch(plan, [&](auto j, auto k) { return launch_group(k_cg64<j, k>, plan, args, st); });
}

cudaError_t launch_cg_mixed(const CgPlan& plan, int grid, const PoissonView& A, const double* b, double* x, double* zp,
                            PcgScalars* sc, double* slots, double rtol, int max_iter, cudaStream_t st)
{
    cudaError_t e = cudaMemsetAsync(slots, 0, plan.planes * kCgPlaneBytes, st);
    if (e != cudaSuccess) return e;
    int smem = plan.smem;
    void* args[] = {(void*)&A, &b, &x, &zp, &sc, &slots, &grid, &rtol, &max_iter, &smem};
    return cg_dispatch(plan, [&](auto j, auto k) { return launch_group(k_cg_mixed<j, k>, plan, args, st); });
}

}  // namespace scdat
