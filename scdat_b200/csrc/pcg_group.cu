// pcg_group.cu -- launches of the one-launch Jacobi-PCG (pcg_group.cuh) on a single system.
#include "pcg_group.cuh"

#include <algorithm>

namespace scdat {

namespace {

template <int KR>
__global__ void __launch_bounds__(kCgMaxThreads, 1)
    k_cg64(const __grid_constant__ PoissonView A, const double* b, double* x, double2* zp, PcgScalars* sc,
           unsigned long long* slots, double rtol, int max_iter, int smem_bytes)
{
    extern __shared__ __align__(16) unsigned char smem[];
    CgGroup g{blockIdx.x, gridDim.x, slots};
    cg_solve64<KR>(g, A, b, x, zp, sc, rtol, max_iter, smem, smem_bytes);
}

template <int KR>
__global__ void __launch_bounds__(kCgMaxThreads, 1)
    k_cg_mixed(const __grid_constant__ PoissonView A, const double* b, double* x, double2* zp, PcgScalars* sc,
               unsigned long long* slots, double rtol, int max_iter, int smem_bytes)
{
    extern __shared__ __align__(16) unsigned char smem[];
    CgGroup g{blockIdx.x, gridDim.x, slots};
    cg_solve_mixed<KR>(g, A, b, x, zp, sc, rtol, max_iter, smem, smem_bytes);
}

// Cooperative launch: the group's blocks wait on one another, so all of them have to be resident.
template <typename K>
cudaError_t launch_group(K kernel, const CgPlan& plan, void** args, cudaStream_t st)
{
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kCgSmemBytes);
    if (e != cudaSuccess) return e;
    return cudaLaunchCooperativeKernel((const void*)kernel, dim3(plan.blocks), dim3(plan.threads), args,
                                       (size_t)plan.smem, st);
}

}  // namespace

CgPlan cg_plan(const int* rows, int n, int nsm, int* blocks_of)
{
    CgPlan plan;
    if (nsm > kCgMaxGroup) nsm = kCgMaxGroup;
    int most = 0;
    for (int k = 0; k < n; ++k) most = std::max(most, rows[k]);
    const bool one_block = most > 256 && most <= kCgMaxThreads;
    for (int kr = 1; kr <= kCgRowsPerThread; ++kr)
        for (int threads = kr == 1 && !one_block ? 256 : kCgMaxThreads; threads <= kCgMaxThreads; threads *= 2) {
            int64_t blocks = 0;
            for (int k = 0; k < n; ++k) {
                const int64_t per = (int64_t)threads * kr;
                blocks_of[k] = (int)((rows[k] + per - 1) / per);
                if (blocks_of[k] < 1) blocks_of[k] = 1;
                blocks += blocks_of[k];
            }
            if (blocks > nsm) continue;
            plan.threads = threads;
            plan.rows_per_thread = kr;
            plan.blocks = (int)blocks;
            const int64_t want = (int64_t)threads * kr * kCgRowSlots * kCgEntryBytes;
            plan.smem = (int)(want < kCgSmemBytes ? want : kCgSmemBytes);
            plan.ok = true;
            return plan;
        }
    return plan;
}

cudaError_t launch_cg64(const CgPlan& plan, const PoissonView& A, const double* b, double* x, double* zp,
                        PcgScalars* sc, double* slots, double rtol, int max_iter, cudaStream_t st)
{
    cudaError_t e = cudaMemsetAsync(slots, 0, kCgSlotBytes, st);
    if (e != cudaSuccess) return e;
    int smem = plan.smem;
    void* args[] = {(void*)&A, &b, &x, &zp, &sc, &slots, &rtol, &max_iter, &smem};
    if (plan.rows_per_thread == 1) return launch_group(k_cg64<1>, plan, args, st);
    if (plan.rows_per_thread == 2) return launch_group(k_cg64<2>, plan, args, st);
    if (plan.rows_per_thread == 3) return launch_group(k_cg64<3>, plan, args, st);
    return launch_group(k_cg64<4>, plan, args, st);
}

cudaError_t launch_cg_mixed(const CgPlan& plan, const PoissonView& A, const double* b, double* x, double* zp,
                            PcgScalars* sc, double* slots, double rtol, int max_iter, cudaStream_t st)
{
    cudaError_t e = cudaMemsetAsync(slots, 0, kCgSlotBytes, st);
    if (e != cudaSuccess) return e;
    int smem = plan.smem;
    void* args[] = {(void*)&A, &b, &x, &zp, &sc, &slots, &rtol, &max_iter, &smem};
    if (plan.rows_per_thread == 1) return launch_group(k_cg_mixed<1>, plan, args, st);
    if (plan.rows_per_thread == 2) return launch_group(k_cg_mixed<2>, plan, args, st);
    if (plan.rows_per_thread == 3) return launch_group(k_cg_mixed<3>, plan, args, st);
    return launch_group(k_cg_mixed<4>, plan, args, st);
}

}  // namespace scdat
