// pcg_group.cuh -- Jacobi-PCG as one launch: a group of co-resident blocks runs the whole solve,
// its rows' CG vectors in registers, its matrix rows in shared memory, two group barriers per
// iteration.  Used by the single-context solves, the CSR entry points (pcg_group.cu) and, one
// group per scenario, by the batched step (batch_field.cu).
//
// What bounds it: the two barriers of an iteration (3.4 us of 5.4 at 137 blocks) and the gathers'
// round trip to L2, not bandwidth.  The systems it takes (up to kCgMaxThreads * kCgRowsPerThread
// rows per SM, 303,104 in all) fit the chip, so the two launches per iteration of the bandwidth
// kernels (field_kern.cuh) were launch gaps and reduction tails, plus a host read every 16
// iterations.  Whole field stages, two launches per iteration against one launch: FP64 33x27x41
// cells 2.14 -> 0.56 ms, 48^3 3.28 -> 1.00, 66^3 6.40 -> 2.61; mixed 40^3 3.27 -> 1.08, 66^3 7.80 -> 3.84.
// Larger systems keep the bandwidth kernels: their rows would no longer fit registers.
//
// The arithmetic is that of field_kern.cuh: FP64 sums and scalars, vectors rounded to V.  Each
// block's part of a dot product is summed by a fixed tree and the blocks' parts in block order, so
// a solve gives the same bits on every run (and in a one-scenario batch, which has the same plan).
#pragma once

#include "field.cuh"

namespace scdat {

constexpr int kCgMaxThreads = 512;                           // one block per SM at most
constexpr int kCgRowsPerThread = 4;                          // most rows a thread holds
constexpr int kCgSmemBytes = 192 * 1024;                     // matrix rows kept per block, at most
constexpr int kCgRowSlots = 16;                              // entries per row kept there (Kuhn meshes: 14)
constexpr int kCgEntryBytes = 12;                            // FP64 value and column
constexpr int kCgMaxGroup = 160;                             // blocks of a group, at most
constexpr int kCgSlotWords = 16;                             // words between barrier slots: a 128-byte line
constexpr size_t kCgSlotBytes = 2 * sizeof(unsigned long long) * kCgSlotWords * kCgMaxGroup;
constexpr unsigned kCgMaxPolls = 1u << 22;                   // bound of a barrier wait (seconds)

// Launch shape of the groups: threads per block, rows per thread, blocks of each group.
struct CgPlan {
    int threads = 0, rows_per_thread = 0, blocks = 0, smem = 0;
    bool ok = false;
};

// A group of g.n blocks of one launch; this block is g.b.  slots: kCgSlotBytes, zero at launch.
struct CgGroup {
    unsigned b, n;
    unsigned long long* slots;
    unsigned epoch = 0;
    bool dead = false;  // a barrier wait ran out: every result is void
};

// A sum in a slot: two 64-bit words of 32 data bits and the barrier's number, so that a reader knows
// each word by itself.
__device__ __forceinline__ void slot_words(double v, unsigned epoch, unsigned long long (&w)[2])
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    w[0] = (b << 32) | epoch;
    w[1] = (b & 0xffffffff00000000ull) | epoch;
}

__device__ __forceinline__ bool slot_sum(const unsigned long long (&w)[2], unsigned epoch, double& v)
{
    v = __longlong_as_double((long long)((w[1] & 0xffffffff00000000ull) | (w[0] >> 32)));
    return (unsigned)w[0] == epoch && (unsigned)w[1] == epoch;
}

// One lane posts NV sums (1 to 3) in a slot.
template <int NV>
__device__ __forceinline__ void slot_post(unsigned long long* slot, unsigned epoch, const double (&s)[NV])
{
    unsigned long long a[2], b[2];
    slot_words(s[0], epoch, a);
    slot_words(NV > 1 ? s[NV > 1 ? 1 : 0] : 0.0, epoch, b);
    if (NV > 2) {
        unsigned long long c[2];
        slot_words(s[NV - 1], epoch, c);
        __stcg(reinterpret_cast<ulonglong2*>(slot) + 2, make_ulonglong2(c[0], c[1]));
    }
    asm volatile("st.relaxed.gpu.global.v4.u64 [%0], {%1, %2, %3, %4};" ::"l"(slot), "l"(a[0]), "l"(a[1]), "l"(b[0]),
                 "l"(b[1])
                 : "memory");
}

// Reads a slot until all its words carry the barrier's number; false when the wait ran out.  One
// 256-bit load brings two sums: 137 blocks 1.2 us for one sum, 2.2 for two with data, against 1.4 and
// 2.8 with a 128-bit load each.
template <int NV>
__device__ __forceinline__ bool slot_wait(const unsigned long long* slot, unsigned epoch, double (&s)[NV])
{
    for (unsigned polls = 0; polls < kCgMaxPolls; ++polls) {
        unsigned long long a[2], b[2];
        asm volatile("ld.relaxed.gpu.global.v4.u64 {%0, %1, %2, %3}, [%4];"
                     : "=l"(a[0]), "=l"(a[1]), "=l"(b[0]), "=l"(b[1])
                     : "l"(slot)
                     : "memory");
        double second;
        bool here = slot_sum(a, epoch, s[0]);
        here = slot_sum(b, epoch, second) && here;
        if (NV > 1) s[NV > 1 ? 1 : 0] = second;
        if (NV > 2) {
            unsigned long long c[2];
            asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];"
                         : "=l"(c[0]), "=l"(c[1]) : "l"(slot + 4) : "memory");
            here = slot_sum(c, epoch, s[NV - 1]) && here;
        }
        if (here) return true;
    }
    return false;
}

// Acquire-release only: __threadfence() is sequentially consistent and costs about twice as much.
__device__ __forceinline__ void fence_acq_rel() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

// Group barrier that also sums: v[k] becomes the sum over every thread of the group.  A block posts
// its part in its slot, a line of its own, and reads every other's: one trip through L2 where an
// arrival counter takes one to arrive, one to poll and one to read the parts.  Alone, for one sum
// without data and two sums with it, 14 blocks 1.0 / 1.7 us, 35 blocks 1.0 / 2.0, 137 blocks
// 1.2 / 2.2 (counter and __threadfence: 2.2 / 2.7, 2.4 / 3.4, 2.7 / 3.4; slots gathered 16 at a
// time by a first block above 32: 1.7 / 3.3 and 2.0 / 3.7).  With DATA, everything a thread of the
// group wrote to global memory before is visible to the others after.
template <int NV, bool DATA>
__device__ __forceinline__ void group_sync_sum(CgGroup& g, double (&v)[NV])
{
    __shared__ double wsum[NV][32];
    __shared__ double psum[NV][kCgMaxGroup / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
        if (lane == 0) wsum[k][warp] = v[k];
    }
    __syncthreads();
    ++g.epoch;
    // two sets of slots in turn: a block may post for the next barrier while another still reads
    unsigned long long* slots = g.slots + (size_t)(g.epoch & 1) * kCgSlotWords * kCgMaxGroup;
    if (warp == 0) {
        double s[NV];
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            s[k] = lane < nw ? wsum[k][lane] : 0.0;
            for (int o = 16; o > 0; o >>= 1) s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
        }
        if (lane == 0) {
            if (g.n == 1) {
#pragma unroll
                for (int k = 0; k < NV; ++k) psum[k][0] = s[k];
            } else {
                if (DATA) fence_acq_rel();
                slot_post<NV>(slots + (size_t)kCgSlotWords * g.b, g.epoch, s);
            }
        }
    }
    int bad = 0;
    if (g.n > 1 && 32u * warp < g.n) {
        const unsigned from = 32u * warp + lane;
        double s[NV];
#pragma unroll
        for (int k = 0; k < NV; ++k) s[k] = 0.0;
        if (from < g.n && !slot_wait<NV>(slots + (size_t)kCgSlotWords * from, g.epoch, s)) bad = 1;
        if (DATA) fence_acq_rel();
        __syncwarp();
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            for (int o = 16; o > 0; o >>= 1) s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
            if (lane == 0) psum[k][warp] = s[k];
        }
    }
    if (__syncthreads_or(bad)) g.dead = true;
    const int np = (int)((g.n + 31) / 32);
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        v[k] = psum[k][0];
        for (int w = 1; w < np; ++w) v[k] += psum[k][w];
    }
}

// This thread's rows of the matrix: the first `width` entries of each in shared memory (entry k of
// slot s at k * slots + s), the others read from the CSR arrays.  FP32 entries are kept as the
// doubles they are used as: converting them, and the gathered vectors, entry by entry cost 1.5 to
// 2 us an iteration.
template <typename V, int KR>
struct CgRows {
    int row[KR];   // -1: none
    int e0[KR], len[KR];
    const int32_t* col;
    const V* val;
    double* sval;
    int32_t* scol;
    int width, slots;
};

template <typename V, int KR>
__device__ __forceinline__ void cg_load_rows(CgRows<V, KR>& A, const CgGroup& g, int R, const int32_t* row_ptr,
                                             const int32_t* col, const V* val, unsigned char* smem, int smem_bytes)
{
    A.slots = blockDim.x * KR;
    A.width = min(kCgRowSlots, smem_bytes / (A.slots * kCgEntryBytes));
    A.sval = reinterpret_cast<double*>(smem);
    A.scol = reinterpret_cast<int32_t*>(A.sval + (size_t)A.width * A.slots);
    A.col = col;
    A.val = val;
#pragma unroll
    for (int j = 0; j < KR; ++j) {
        const int i = (g.b + j * g.n) * blockDim.x + threadIdx.x;
        A.row[j] = i < R ? i : -1;
        A.e0[j] = 0;
        A.len[j] = 0;
        if (i < R) {
            A.e0[j] = __ldg(row_ptr + i);
            A.len[j] = __ldg(row_ptr + i + 1) - A.e0[j];
            // a row shorter than the width ends in zero entries on its own column
            const int slot = j * blockDim.x + threadIdx.x;
            for (int k = 0; k < A.width; ++k) {
                const bool on = k < A.len[j];
                A.sval[k * A.slots + slot] = on ? (double)__ldg(val + A.e0[j] + k) : 0.0;
                A.scol[k * A.slots + slot] = on ? __ldg(col + A.e0[j] + k) : i;
            }
        }
    }
    // each thread reads only its own slots: no barrier
}

// s + sum over row j's entries of val * x(col), in the row's order; the gathers of a batch of
// entries (a whole row, mostly) are in flight together.
template <typename V, int KR, typename F>
__device__ __forceinline__ double cg_row_apply(const CgRows<V, KR>& A, int j, double s, F&& x)
{
    const double* v = A.sval + j * blockDim.x + threadIdx.x;
    const int32_t* c = A.scol + j * blockDim.x + threadIdx.x;
    if (A.width == kCgRowSlots) {
        double xv[kCgRowSlots];
#pragma unroll
        for (int k = 0; k < kCgRowSlots; ++k) xv[k] = x(c[k * A.slots]);
#pragma unroll
        for (int k = 0; k < kCgRowSlots; ++k) s += v[k * A.slots] * xv[k];
    } else {
        for (int k = 0; k < A.width; ++k) s += v[k * A.slots] * x(c[k * A.slots]);
    }
    for (int k = A.width; k < A.len[j]; ++k) s += (double)__ldg(A.val + A.e0[j] + k) * x(__ldg(A.col + A.e0[j] + k));
    return s;
}

// A vector element as the solve stores it.
template <typename V>
__device__ __forceinline__ double as_stored(double v)
{
    return (double)(V)v;
}

// The CG loop on V vectors, carried as doubles that hold V values.  In: x, r, z of this thread's
// rows, with (z, 0) in zp (a DATA barrier has passed since).  zp holds each row's z and last
// direction side by side, so the mat-vec builds a column's new direction z + beta p from one load;
// it is written once an iteration, between the two barriers the mat-vec does not touch it in, and read
// through L1, which the second barrier's fences empty (FP64 field stage of 117 rows 95 -> 79 us,
// 33x27x41 cells 569 -> 558; a batch of 8 with two rows a thread, four steps, 7.01 -> 6.94 ms).
struct CgScalars {
    double rz, rz_prev, rr, thr2;
    int iter, max_iter;
    bool done;
};

template <typename V, int KR>
__device__ __forceinline__ void cg_iterate(CgGroup& g, const CgRows<V, KR>& A, const double (&diag)[KR],
                                           const double (&dinv)[KR], double (&x)[KR], double (&r)[KR],
                                           double (&z)[KR], double2* zp, CgScalars& c)
{
    double p[KR];
#pragma unroll
    for (int j = 0; j < KR; ++j) p[j] = 0.0;
    while (!c.done && !g.dead) {
        const double beta = c.iter == 0 ? 0.0 : c.rz / c.rz_prev;
        double q[KR], acc[1] = {0.0};
#pragma unroll
        for (int j = 0; j < KR; ++j) {
            q[j] = 0.0;
            if (A.row[j] < 0) continue;
            const double pi = z[j] + beta * p[j];
            const double s = cg_row_apply(A, j, diag[j] * pi, [&](int c0) {
                const double2 n = zp[c0];  // by L1: a block's rows are neighbours
                return n.x + beta * n.y;
            });
            p[j] = as_stored<V>(pi);
            q[j] = as_stored<V>(s);
            acc[0] += pi * s;
        }
        group_sync_sum<1, false>(g, acc);
        const double pq = acc[0];
        const double alpha = pq > 0.0 ? c.rz / pq : 0.0;
        double dots[2] = {0.0, 0.0};
#pragma unroll
        for (int j = 0; j < KR; ++j) {
            if (A.row[j] < 0) continue;
            const double ri = r[j] - alpha * q[j];
            const double zi = ri * dinv[j];
            x[j] = as_stored<V>(x[j] + alpha * p[j]);
            r[j] = as_stored<V>(ri);
            z[j] = as_stored<V>(zi);
            __stcg(zp + A.row[j], make_double2(z[j], p[j]));
            dots[0] += ri * zi;
            dots[1] += ri * ri;
        }
        group_sync_sum<2, true>(g, dots);
        c.rz_prev = c.rz;
        c.rz = dots[0];
        c.rr = dots[1];
        c.iter += 1;
        if (c.rr <= c.thr2 || c.iter >= c.max_iter || !(pq > 0.0)) c.done = true;
    }
}

// FP64 CG from x (k_pcg_init + the k_pcg_spmv / k_pcg_update loop); zp: 2 R values.
template <int KR>
__device__ __forceinline__ void cg_solve64(CgGroup g, const PoissonView& P, const double* b, double* xg, double2* zp,
                                           PcgScalars* sc, double rtol, int max_iter, unsigned char* smem,
                                           int smem_bytes)
{
    CgRows<double, KR> A;
    cg_load_rows(A, g, P.R, P.row_ptr, P.col, P.val, smem, smem_bytes);
    double x[KR], r[KR], z[KR], diag[KR], dinv[KR], acc[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int j = 0; j < KR; ++j) {
        x[j] = r[j] = z[j] = diag[j] = dinv[j] = 0.0;
        const int i = A.row[j];
        if (i < 0) continue;
        diag[j] = P.diag[i];
        dinv[j] = P.dinv ? P.dinv[i] : 1.0 / diag[j];
        x[j] = xg[i];
        const double bi = b[i];
        r[j] = bi - cg_row_apply(A, j, diag[j] * x[j], [&](int c0) { return __ldcg(xg + c0); });
        z[j] = r[j] * dinv[j];
        __stcg(zp + i, make_double2(z[j], 0.0));
        acc[0] += r[j] * z[j];
        acc[1] += r[j] * r[j];
        acc[2] += bi * bi;
    }
    group_sync_sum<3, true>(g, acc);
    CgScalars c{};
    c.rz = acc[0];
    c.rz_prev = 1.0;
    c.rr = acc[1];
    c.thr2 = rtol * rtol * (acc[2] > 0.0 ? acc[2] : 1.0);
    c.max_iter = max_iter;
    c.done = c.rr <= c.thr2 || max_iter <= 0;
    cg_iterate<double, KR>(g, A, diag, dinv, x, r, z, zp, c);
#pragma unroll
    for (int j = 0; j < KR; ++j)
        if (A.row[j] >= 0) xg[A.row[j]] = x[j];
    if (g.b == 0 && threadIdx.x == 0) {
        sc->rz = c.rz;
        sc->rz_prev = c.rz_prev;
        sc->rr = c.rr;
        sc->bb = acc[2];
        sc->thr2 = c.thr2;
        sc->iter = c.iter;
        sc->done = g.dead ? -1 : 1;
    }
}

// The precision form's solve: FP32 CG for the correction inside FP64 refinement (the loop of
// run_pcg_mixed in capi.cu), all passes in this call.  sc: rr, bb, iter (inner iterations in all)
// and outer (passes) out.
template <int KR>
__device__ __forceinline__ void cg_solve_mixed(CgGroup g, const PoissonView& P, const double* b, double* xg,
                                               double2* zp, PcgScalars* sc, double rtol, int max_iter,
                                               unsigned char* smem, int smem_bytes)
{
    CgRows<float, KR> A;
    cg_load_rows(A, g, P.R, P.row_ptr, P.col, P.valf, smem, smem_bytes);
    double x[KR], diag[KR], dinv[KR];
#pragma unroll
    for (int j = 0; j < KR; ++j) {
        x[j] = diag[j] = dinv[j] = 0.0;
        if (A.row[j] < 0) continue;
        x[j] = xg[A.row[j]];
        diag[j] = (double)P.diagf[A.row[j]];
        dinv[j] = (double)P.dinvf[A.row[j]];
    }
    int iters = 0, outer = 0;
    double norm[2];
    for (;; ++outer) {
        double e[KR], r[KR], z[KR], acc[2] = {0.0, 0.0};
        norm[0] = norm[1] = 0.0;
#pragma unroll
        for (int j = 0; j < KR; ++j) {
            e[j] = r[j] = z[j] = 0.0;
            const int i = A.row[j];
            if (i < 0) continue;
            // the FP64 matrix's values are read: two to four of these against an iteration each time
            double s = P.diag[i] * x[j];
            const double* val = P.val + A.e0[j];
            const int32_t* col = P.col + A.e0[j];
#pragma unroll 4
            for (int k = 0; k < A.len[j]; ++k) s += __ldg(val + k) * __ldcg(xg + __ldg(col + k));
            const double bi = b[i], ri = bi - s;
            norm[0] += ri * ri;
            norm[1] += bi * bi;
            // the start of A e = r from e = 0
            r[j] = as_stored<float>(ri);
            const double zf = r[j] * dinv[j];
            z[j] = as_stored<float>(zf);
            __stcg(zp + i, make_double2(z[j], 0.0));
            acc[0] += r[j] * zf;
            acc[1] += r[j] * r[j];
        }
        group_sync_sum<2, true>(g, norm);
        const double bb = norm[1] > 0.0 ? norm[1] : 1.0;
        if (g.dead || norm[0] <= rtol * rtol * bb || iters >= max_iter || outer == kMaxRefinePasses) break;
        group_sync_sum<2, false>(g, acc);
        // to the tolerance this pass needs
        const double rt = inner_rtol(norm[0], bb, rtol);
        CgScalars c{};
        c.rz = acc[0];
        c.rz_prev = 1.0;
        c.rr = acc[1];
        c.thr2 = rt * rt * (acc[1] > 0.0 ? acc[1] : 1.0);
        c.max_iter = max(1, max_iter - iters);
        c.done = c.rr <= c.thr2;
        cg_iterate<float, KR>(g, A, diag, dinv, e, r, z, zp, c);
        iters += c.iter;
#pragma unroll
        for (int j = 0; j < KR; ++j) {
            if (A.row[j] < 0) continue;
            x[j] += e[j];
            __stcg(xg + A.row[j], x[j]);
        }
        double none[1] = {0.0};
        group_sync_sum<1, true>(g, none);  // x is read by the other blocks' residuals
    }
    if (g.b == 0 && threadIdx.x == 0) {
        sc->rr = norm[0];
        sc->bb = norm[1];
        sc->iter = iters;
        sc->outer = outer;
        sc->done = g.dead ? -1 : 1;
    }
}

// Launch shape for groups of the given row counts on nsm SMs: one block per SM at most, as many as
// the rows fill (a row more per thread costs an iteration 0.8 to 1.6 us, 102 more blocks 1 us of
// barrier: 33x27x41 cells, 35k rows, first barrier form, 137 blocks of 256 777 us, 69 of 512 833, 35
// of 512 with two rows a thread 955), then more rows per thread, the same for every group (a batch of 8 with one row
// a thread in its largest scenario and more in the others 7.33 ms, two in each 7.07); up to 512 rows one
// block, whose barriers stay in the SM (FP64 field stage of 335 rows 151 -> 108 us, 504 rows 153 -> 127;
// 992 rows two a thread in one block 199, in four blocks 177); !ok when that does not fit.
// blocks_of: blocks of each group.
CgPlan cg_plan(const int* rows, int n, int nsm, int* blocks_of);

// One system: queues the solve on st.  zp: 2 R values; slots: kCgSlotBytes; results in sc (done < 0:
// a barrier wait ran out).
cudaError_t launch_cg64(const CgPlan& plan, const PoissonView& A, const double* b, double* x, double* zp,
                        PcgScalars* sc, double* slots, double rtol, int max_iter, cudaStream_t st);
cudaError_t launch_cg_mixed(const CgPlan& plan, const PoissonView& A, const double* b, double* x, double* zp,
                            PcgScalars* sc, double* slots, double rtol, int max_iter, cudaStream_t st);

}  // namespace scdat
