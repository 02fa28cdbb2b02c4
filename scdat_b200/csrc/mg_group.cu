// mg_group.cu -- the multigrid-preconditioned CG as one cooperative launch per solve.
//
// An iteration is 25 to 32 dependent passes over levels of 250k rows down to a few hundred, most
// of them shorter than a launch, and the host read the convergence flag every second iteration.
// Here one block per SM keeps all of it in one launch: a barrier between passes instead of a
// launch, the first damped-Jacobi sweep of a level written by the pass that makes its right-hand
// side, matrix and transfer rows side by side (coalesced, fourteen entries of a row in flight,
// since 16 warps per SM hide little; two rows at once spilled and took 1.34 ms for 1.28).  The
// arithmetic is mg.cu's: sweeps and transfers in V, the CG's mat-vec and scalars in FP64.  At 64^3
// cells in FP32 a field solve takes 1.28 ms, by launches 2.09 ms.  What bounds it: some 25 barriers
// of 1.2 us and more an iteration, each behind a chain of three dependent reads (column, vector,
// sum); the finest level's passes, 28 MB of rows from L2, are half of an iteration.
#include "mg_group.cuh"

namespace scdat {

namespace {

// The column of a filling entry is the row's last one, in cache beside it: with column 0 in all of
// them the finest prolongation, most of whose rows are short, took 18 us on that one line (field
// solve at 64^3 cells 1.52 ms, not 1.43).
template <typename S, typename V>
__global__ void k_csr_to_ell(int R, int width, const int32_t* __restrict__ ptr, const int32_t* __restrict__ col,
                             const S* __restrict__ val, V* __restrict__ ev, int32_t* __restrict__ ec)
{
    for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < (int64_t)width * R;
         g += (int64_t)gridDim.x * blockDim.x) {
        const int k = (int)(g / R), i = (int)(g % R);
        const int e = ptr[i] + k, end = ptr[i + 1];
        ev[g] = e < end ? (V)val[e] : (V)0;
        ec[g] = ptr[i] < end ? col[e < end ? e : end - 1] : 0;
    }
}

// s + sum over row i of val * x(col), in the row's order, summed in S; B entries in flight, the next
// ones' columns beside them.  The width is a batch at least.
template <int B, typename S, typename V>
__device__ __forceinline__ S ell_row(const EllDev<V>& A, int i, S s, const V* x)
{
    int32_t c[B];
#pragma unroll
    for (int k = 0; k < B; ++k) c[k] = __ldg(A.col + (size_t)k * A.pad + i);
    for (int k0 = 0; k0 < A.width; k0 += B) {
        V v[B], y[B];
#pragma unroll
        for (int k = 0; k < B; ++k) {
            y[k] = x[c[k]];
            v[k] = __ldg(A.val + (size_t)(k0 + k) * A.pad + i);
        }
        if (k0 + B < A.width)
#pragma unroll
            for (int k = 0; k < B; ++k) c[k] = __ldg(A.col + (size_t)(k0 + B + k) * A.pad + i);
#pragma unroll
        for (int k = 0; k < B; ++k) s += (S)v[k] * (S)y[k];
    }
    return s;
}

// f(row) over this thread's rows of a level: neighbouring rows in one block, but a level of fewer
// rows than threads spread over all blocks by warps (on the first blocks alone its passes at 64^3
// cells took 1.05 times the whole solve).
template <typename F>
__device__ __forceinline__ void each_row(int R, const CgGroup& g, F&& f)
{
    const int step = g.n * blockDim.x;
    int i = g.b * blockDim.x + threadIdx.x;
    if (R <= step) i = ((threadIdx.x >> 5) * g.n + g.b) * 32 + (threadIdx.x & 31);
    for (; i < R; i += step) f(i);
}

__device__ __forceinline__ void barrier(CgGroup& g)
{
    double none[1] = {0.0};
    group_sync_sum<1, true>(g, none);
}

// xo = xi + omega D^-1 (b - A xi); with DOT this thread's part of b . xo
template <typename V, bool DOT>
__device__ __forceinline__ double sweep(const MgGroupLevel<V>& L, const CgGroup& g, const V* b, const V* xi, V* xo)
{
    double dot = 0.0;
    each_row(L.R, g, [&](int i) {
        const V xv = __ldcg(xi + i), bi = __ldcg(b + i);
        const V v = xv + L.omega * L.dinv[i] * (bi - ell_row<kMgEllBatch>(L.A, i, L.diag[i] * xv, xi));
        __stcg(xo + i, v);
        if (DOT) dot += (double)bi * (double)v;
    });
    return dot;
}

// One V-cycle z = M r with r in L[0]'s right-hand side `b0` and its first sweep in L[0].xa (both
// visible); returns this thread's part of r . z (the caller's next barrier sums it).
template <typename V>
__device__ __forceinline__ double vcycle(const MgGroupPlan<V>& mg, const MgGroupLevel<V>* lv, CgGroup& g, const V* b0,
                                         V* z)
{
    const int top = mg.levels - 1;
    for (int l = 0; l < top; ++l) {
        const MgGroupLevel<V>& L = lv[l];
        const MgGroupLevel<V>& C = lv[l + 1];
        const V* b = l == 0 ? b0 : L.b;
        sweep<V, false>(L, g, b, L.xa, L.xb);
        barrier(g);
        each_row(L.R, g, [&](int i) {
            __stcg(L.res + i, __ldcg(b + i) - ell_row<kMgEllBatch>(L.A, i, L.diag[i] * __ldcg(L.xb + i), L.xb));
        });
        barrier(g);
        const bool last = l + 1 == top;
        each_row(C.R, g, [&](int i) {
            const V s = ell_row<kMgEllBatch>(L.Rt, i, (V)0, L.res);
            __stcg(C.b + i, s);
            if (!last) __stcg(C.xa + i, C.omega * C.dinv[i] * s);
        });
        barrier(g);
    }
    {
        // the coarsest level: one warp per row of the dense inverse
        const MgGroupLevel<V>& C = lv[top];
        const int R = C.R, lane = threadIdx.x & 31, warps = g.n * (blockDim.x >> 5);
        for (int row = (threadIdx.x >> 5) * g.n + g.b; row < R; row += warps) {
            const V* a = mg.cinv + (size_t)row * R;
            V s = 0;
#pragma unroll 8
            for (int j = lane; j < R; j += 32) s += __ldg(a + j) * __ldcg(C.b + j);
            for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
            if (lane == 0) __stcg(C.xo + row, s);
        }
        barrier(g);
    }
    for (int l = top - 1;; --l) {
        const MgGroupLevel<V>& L = lv[l];
        const V* xc = lv[l + 1].xo;
        const V* b = l == 0 ? b0 : L.b;
        each_row(L.R, g, [&](int i) {
            __stcg(L.xb + i, __ldcg(L.xb + i) + ell_row<kMgEllTransfer>(L.P, i, (V)0, xc));
        });
        barrier(g);
        sweep<V, false>(L, g, b, L.xb, L.xa);
        barrier(g);
        if (l == 0) return sweep<V, true>(L, g, b, L.xa, z);
        sweep<V, false>(L, g, b, L.xa, L.xo);
        barrier(g);
    }
}

template <typename V>
__global__ void __launch_bounds__(kMgGroupThreads, 1)
    k_mgpcg_group(MgGroupPlan<V> mg, const V* b, V* x, V* r, V* z, V* p, V* q, int zero_start, double rtol, int max_iter,
                  PcgScalars* sc, unsigned long long* slots)
{
    __shared__ MgGroupLevel<V> lv[kMgMaxLevels];  // the barriers' fences would drop it from L1 every pass
    for (int w = threadIdx.x; w < (int)(mg.levels * sizeof(lv[0]) / sizeof(int)); w += blockDim.x)
        reinterpret_cast<int*>(lv)[w] = reinterpret_cast<const int*>(mg.lv)[w];
    __syncthreads();
    CgGroup g{blockIdx.x, gridDim.x, slots};
    const MgGroupLevel<V>& L = lv[0];
    // the residual and the first sweep of the first cycle
    double acc[2] = {0.0, 0.0};
    each_row(L.R, g, [&](int i) {
        const double bi = (double)b[i];
        const double ax =
            zero_start ? 0.0 : ell_row<kMgEllBatch>(L.A, i, (double)L.diag[i] * (double)__ldcg(x + i), x);
        const double ri = bi - ax;
        const V rv = (V)ri;
        __stcg(r + i, rv);
        __stcg(L.xa + i, L.omega * L.dinv[i] * rv);
        if (zero_start) x[i] = (V)0;
        acc[0] += ri * ri;
        acc[1] += bi * bi;
    });
    group_sync_sum<2, true>(g, acc);
    double rr = acc[0], rz_prev = 1.0;
    const double bb = acc[1], thr2 = rtol * rtol * (bb > 0.0 ? bb : 1.0);
    bool done = rr <= thr2 || max_iter <= 0;
    int iter = 0;
    while (!done && !g.dead) {
        double rz[1] = {vcycle<V>(mg, lv, g, r, z)};
        group_sync_sum<1, true>(g, rz);
        const V beta = iter == 0 ? (V)0 : (V)(rz[0] / rz_prev);
        each_row(L.R, g, [&](int i) {
            const V zi = __ldcg(z + i);
            __stcg(p + i, iter == 0 ? zi : zi + beta * __ldcg(p + i));
        });
        barrier(g);
        double pq[1] = {0.0};
        each_row(L.R, g, [&](int i) {
            const double pv = (double)__ldcg(p + i);
            const double s = ell_row<kMgEllBatch>(L.A, i, (double)L.diag[i] * pv, p);
            __stcg(q + i, (V)s);
            pq[0] += pv * s;
        });
        group_sync_sum<1, false>(g, pq);
        const double alpha = pq[0] > 0.0 ? rz[0] / pq[0] : 0.0;
        double rn[1] = {0.0};
        each_row(L.R, g, [&](int i) {
            const double ri = (double)__ldcg(r + i) - alpha * (double)__ldcg(q + i);
            const V rv = (V)ri;
            x[i] = (V)((double)x[i] + alpha * (double)__ldcg(p + i));
            __stcg(r + i, rv);
            __stcg(L.xa + i, L.omega * L.dinv[i] * rv);
            rn[0] += ri * ri;
        });
        group_sync_sum<1, true>(g, rn);
        rz_prev = rz[0];
        rr = rn[0];
        ++iter;
        done = rr <= thr2 || iter >= max_iter || !(pq[0] > 0.0);
    }
    if (g.b == 0 && threadIdx.x == 0) {
        sc->rr = rr;
        sc->bb = bb;
        sc->thr2 = thr2;
        sc->iter = iter;
        sc->done = g.dead ? -1 : 1;
    }
}

}  // namespace

template <typename S, typename V>
void launch_csr_to_ell(int R, int width, const int32_t* ptr, const int32_t* col, const S* val, V* ell_val,
                       int32_t* ell_col, cudaStream_t st)
{
    k_csr_to_ell<S, V><<<148 * 8, 256, 0, st>>>(R, width, ptr, col, val, ell_val, ell_col);
}

template <typename V>
cudaError_t launch_mgpcg_group(const MgGroupPlan<V>& mg, const V* b, V* x, V* r, V* z, V* p, V* q, bool zero_start,
                               double rtol, int max_iter, PcgScalars* sc, double* slots, cudaStream_t st)
{
    cudaError_t e = cudaMemsetAsync(slots, 0, kCgSlotBytes, st);
    if (e != cudaSuccess) return e;
    MgGroupPlan<V> plan = mg;
    int zs = zero_start ? 1 : 0;
    void* args[] = {&plan, &b, &x, &r, &z, &p, &q, &zs, &rtol, &max_iter, &sc, &slots};
    return cg_launch((const void*)k_mgpcg_group<V>, mg.blocks, kMgGroupThreads, args, 0, st);
}

template void launch_csr_to_ell<float, float>(int, int, const int32_t*, const int32_t*, const float*, float*, int32_t*, cudaStream_t);
template void launch_csr_to_ell<float, double>(int, int, const int32_t*, const int32_t*, const float*, double*,
                                               int32_t*, cudaStream_t);
template void launch_csr_to_ell<double, float>(int, int, const int32_t*, const int32_t*, const double*, float*, int32_t*, cudaStream_t);
template void launch_csr_to_ell<double, double>(int, int, const int32_t*, const int32_t*, const double*, double*,
                                                int32_t*, cudaStream_t);
template cudaError_t launch_mgpcg_group<float>(const MgGroupPlan<float>&, const float*, float*, float*, float*, float*,
                                               float*, bool, double, int, PcgScalars*, double*, cudaStream_t);
template cudaError_t launch_mgpcg_group<double>(const MgGroupPlan<double>&, const double*, double*, double*, double*,
                                                double*, double*, bool, double, int, PcgScalars*, double*,
                                                cudaStream_t);

}  // namespace scdat
