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
// cells 2.13 -> 0.54 ms, 48^3 3.30 -> 1.04, 64x66x65 6.29 -> 3.28; mixed 33x27x41 2.52 -> 0.67, 42^3 3.93
// -> 1.15, 64x66x65 7.48 -> 4.03.
// Larger systems keep the bandwidth kernels: their rows would no longer fit registers.
//
// The arithmetic is that of field_kern.cuh, bit for bit: FP64 sums and scalars, vectors rounded to V,
// and every dot product summed in the order of its block_sum and last_block.  A virtual block of 256
// threads stands for a block of the launched form: the same rows, the same tree over its warps, and the
// same tree over the blocks' parts; the rounding is spelled out, since the compiler may contract
// a * b + c * d in two ways.  So a solve, of a context alone or in a batch, gives the bits the
// launched form gives (a plasma that is unstable on its grid magnifies a last-bit change of the
// potential to 1e-3 within a few steps).
#pragma once

#include "field.cuh"

#include <type_traits>

namespace scdat {

constexpr int kCgMaxThreads = 512;                           // one block per SM at most
constexpr int kCgRowsPerThread = 4;                          // most rows a thread holds
constexpr int kCgSmemBytes = 192 * 1024;                     // matrix rows kept per block, at most
constexpr int kCgRowSlots = 16;                              // entries per row kept there (Kuhn meshes: 14)
constexpr int kCgEntryBytes = 12;                            // FP64 value and column
constexpr int kCgMaxGroup = 160;                             // blocks of a group, at most
constexpr int kCgSlotWords = 16;                             // words between barrier slots: a 128-byte line
constexpr int kCgVirtual = 256;                              // threads of a virtual block
constexpr int kCgVirtualWarps = kCgVirtual / 32;
// a plane of slots, a line per block in each of two sets; blocks that post more than 8 sums use two
constexpr size_t kCgPlaneWords = 2 * (size_t)kCgSlotWords * kCgMaxGroup;
constexpr size_t kCgPlaneBytes = kCgPlaneWords * sizeof(unsigned long long);
constexpr size_t kCgSlotBytes = 2 * kCgPlaneBytes;
constexpr unsigned kCgMaxPolls = 1u << 22;                   // bound of a barrier wait (seconds)

// Launch shape of the groups: threads per block, virtual threads of each and rows of a virtual thread
// (rows_per_thread together), blocks of all groups, planes of barrier slots.
struct CgPlan {
    int threads = 0, virt = 0, rounds = 0, rows_per_thread = 0, blocks = 0, smem = 0, planes = 0;
    bool ok = false;
};

// A group of g.n blocks of one launch; this block is g.b.  vgrid: blocks of 256 threads the launched
// form gives the system (rows further than vgrid * 256 apart belong to one thread).  slots: zero at
// launch, the planes in use.
struct CgGroup {
    unsigned b, n;
    unsigned long long* slots;
    unsigned vgrid = 0;
    unsigned epoch = 0;
    bool dead = false;  // a barrier wait ran out: every result is void, and this block posts nothing more
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

// One lane posts two sums side by side.
__device__ __forceinline__ void slot_post(unsigned long long* at, unsigned epoch, double s0, double s1)
{
    unsigned long long a[2], b[2];
    slot_words(s0, epoch, a);
    slot_words(s1, epoch, b);
    asm volatile("st.relaxed.gpu.global.v4.u64 [%0], {%1, %2, %3, %4};" ::"l"(at), "l"(a[0]), "l"(a[1]), "l"(b[0]),
                 "l"(b[1])
                 : "memory");
}

// Reads them once; true when all four words carry the barrier's number.  One 256-bit load: 137 blocks
// 1.2 us for one sum, 2.2 for two with data, against 1.4 and 2.8 with a 128-bit load each.
__device__ __forceinline__ bool slot_read(const unsigned long long* at, unsigned epoch, double& s0, double& s1)
{
    unsigned long long a[2], b[2];
    asm volatile("ld.relaxed.gpu.global.v4.u64 {%0, %1, %2, %3}, [%4];"
                 : "=l"(a[0]), "=l"(a[1]), "=l"(b[0]), "=l"(b[1])
                 : "l"(at)
                 : "memory");
    const bool here = slot_sum(a, epoch, s0);
    return slot_sum(b, epoch, s1) && here;
}

// Acquire-release only: __threadfence() is sequentially consistent and costs about twice as much.
__device__ __forceinline__ void fence_acq_rel() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

// The current barrier's slots: two sets in turn, since a block may post for the next barrier while
// another still reads.
__device__ __forceinline__ unsigned long long* slot_set(const CgGroup& g)
{
    return g.slots + (g.epoch & 1) * (kCgPlaneWords / 2);
}

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
    static_assert(NV == 1 || NV == 2, "one or two sums");
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
    unsigned long long* slots = slot_set(g);
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
            } else if (!g.dead) {
                if (DATA) fence_acq_rel();
                slot_post(slots + (size_t)kCgSlotWords * g.b, g.epoch, s[0], NV > 1 ? s[NV - 1] : 0.0);
            }
        }
    }
    int bad = 0;
    if (g.n > 1 && !g.dead && 32u * warp < g.n) {
        const unsigned from = 32u * warp + lane;
        double s[NV];
#pragma unroll
        for (int k = 0; k < NV; ++k) s[k] = 0.0;
        if (from < g.n) {
            bad = 1;
            double s0 = 0.0, s1 = 0.0;
            for (unsigned polls = 0; bad && polls < kCgMaxPolls; ++polls)
                if (slot_read(slots + (size_t)kCgSlotWords * from, g.epoch, s0, s1)) bad = 0;
            s[0] = s0;
            if (NV > 1) s[NV - 1] = s1;
        }
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

// The lane's part of the sums over a warp of M values (a power of two, 8 at most): afterwards a[0] of
// lane l is the sum of value l / (32 / M).  Lanes are paired as in block_sum's shuffles (l and l + 16,
// then l + 8, ...), so every sum has its bits; the first steps halve the values instead of repeating
// the exchange for each.
template <int M>
__device__ __forceinline__ void warp_sums(double (&a)[M])
{
    const int lane = threadIdx.x & 31;
    int n = M;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        if (n > 1) {
            n >>= 1;
            const bool up = (lane & o) != 0;
#pragma unroll
            for (int k = 0; k < n; ++k) {
                const double send = up ? a[k] : a[k + n], keep = up ? a[k + n] : a[k];
                a[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
        } else {
            a[0] += __shfl_xor_sync(0xffffffffu, a[0], o);
        }
    }
}

__host__ __device__ constexpr int pow2_from(int n) { return n <= 1 ? 1 : 2 * pow2_from((n + 1) / 2); }

template <int J>
struct DotsShared {
    double wsum[pow2_from(2 * J)][kCgMaxThreads / 32];  // of a warp
    double part[2][2 * J * kCgMaxGroup];                // of a virtual block
    double sum[2];
};

// one for all barriers of a kernel
template <int J>
__device__ __forceinline__ DotsShared<J>& dots_shared()
{
    __shared__ DotsShared<J> s;
    return s;
}

// Group barrier with NV dot products (1 or 2) of J virtual threads per thread: in[k][j] is dot k of
// this thread's virtual thread j; v[k] becomes the sum over the group in the launched form's order
// (see the head of the file).  A block posts the parts of its virtual blocks and reads all of them, and
// one warp a dot does last_block's tree.  Against parts of whole blocks in any order, field stages
// of up to 70k rows took -20 to +10 %, FP64 ones of 100k and 260k rows +5 and +29 %.
template <int NV, int J, bool DATA>
__device__ __forceinline__ void group_sync_dots(CgGroup& g, const double (&in)[NV][J], double (&v)[NV])
{
    static_assert(NV == 1 || NV == 2, "one or two sums");
    constexpr int M = pow2_from(NV * J);
    DotsShared<J>& sh = dots_shared<J>();
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned h = blockDim.x > kCgVirtual ? 1u : 0u;    // log2 of a block's halves
    const unsigned per = (unsigned)J << h, nv = g.n * per;   // virtual blocks: of a block, in all
    double a[M];
#pragma unroll
    for (int k = 0; k < M; ++k) a[k] = k < NV * J ? in[k / J][k % J] : 0.0;
    warp_sums<M>(a);
    if (lane % (32 / M) == 0) sh.wsum[lane / (32 / M)][warp] = a[0];
    __syncthreads();
    ++g.epoch;
    unsigned long long* slots = slot_set(g);
    // place of virtual block e's parts, in the line of its block
    const auto unit_at = [&](unsigned e) {
        const unsigned b = (e >> h) / J, u = e - b * per;
        return slots + (u >> 2) * kCgPlaneWords + kCgSlotWords * b + 4 * (u & 3);
    };
    double t[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) t[k] = 0.0;
    if (warp == 0) {
        // lane u: the parts of this block's u-th virtual block (the other lanes compute the last one's,
        // so that the warp stays together: with one lane apart it met again at every shuffle below,
        // 1.2 us a barrier)
        const unsigned u = min(lane, per - 1), j = u >> h, half = u & h;
#pragma unroll
        for (int w = 0; w < kCgVirtualWarps; ++w)
#pragma unroll
            for (int k = 0; k < NV; ++k) t[k] += sh.wsum[k * J + j][half * kCgVirtualWarps + w];
        if (lane >= per)
#pragma unroll
            for (int k = 0; k < NV; ++k) t[k] = 0.0;
        if (g.n > 1 && !g.dead && lane < per) {
            if (DATA) fence_acq_rel();
            slot_post(unit_at(g.b * per + u), g.epoch, t[0], NV > 1 ? t[NV - 1] : 0.0);
        }
        __syncwarp();
    }
    int bad = 0;
    if (g.n > 1) {
        // Every thread reads parts, two in flight; neighbours those of one block, so that a block's line
        // is one request an SM (148 SMs reading four parts of each line apart took 3 us more).
        constexpr int kReads = J <= 2 ? J : J - 1;
        static_assert(kReads * kCgMaxThreads >= 2 * J * kCgMaxGroup && kCgVirtual >= kCgMaxGroup, "every part is read");
#pragma unroll 1
        for (int r0 = 0; r0 < kReads; r0 += 2) {
            const unsigned e0 = threadIdx.x + r0 * blockDim.x, e1 = e0 + blockDim.x;
            if (e0 - lane >= nv) break;
            const bool on0 = e0 < nv, on1 = kReads > 1 && e1 < nv;
            double m0[2] = {0.0, 0.0}, m1[2] = {0.0, 0.0};
            int wait = g.dead ? 0 : 1;
            for (unsigned polls = 0; wait && polls < kCgMaxPolls; ++polls) {
                bool here = true;
                if (on0) here = slot_read(unit_at(e0), g.epoch, m0[0], m0[1]);
                if (kReads > 1 && on1) here = slot_read(unit_at(e1), g.epoch, m1[0], m1[1]) && here;
                if (here) wait = 0;
            }
            bad |= wait;
#pragma unroll
            for (int k = 0; k < NV; ++k) {
                if (on0) sh.part[k][e0] = m0[k];
                if (kReads > 1 && on1) sh.part[k][e1] = m1[k];
            }
        }
        if (DATA) fence_acq_rel();
        __syncthreads();
        // thread t of last_block's 256 adds the parts t, t + 256, ...; the tree's upper levels are
        // additions in a lane
        if (warp < NV) {
            const double* part = sh.part[warp];
            double m[8];
#pragma unroll
            for (unsigned i = 0; i < 8; ++i) m[i] = 32 * i + lane < nv ? part[32 * i + lane] : 0.0;
            for (unsigned e0 = 256; e0 < nv; e0 += 256)
#pragma unroll
                for (unsigned i = 0; i < 8; ++i)
                    if (e0 + 32 * i + lane < nv) m[i] += part[e0 + 32 * i + lane];
            double s[1] = {((m[0] + m[4]) + (m[2] + m[6])) + ((m[1] + m[5]) + (m[3] + m[7]))};
            warp_sums<1>(s);
            if (lane == 0) sh.sum[warp] = s[0];
        }
    } else if (warp == 0) {
        warp_sums<NV>(t);
        if (lane % (32 / NV) == 0) sh.sum[lane / (32 / NV)] = t[0];
    }
    if (__syncthreads_or(bad)) g.dead = true;
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = sh.sum[k];
}

// This thread's rows of the matrix: the first `width` entries of each in shared memory (entry k of
// slot s at k * slots + s), the others read from the CSR arrays.  FP32 entries are kept as the
// doubles they are used as: converting them, and the gathered vectors, entry by entry cost 1.5 to
// 2 us an iteration.
template <typename V, int J, int K>
struct CgRows {
    static constexpr int KR = J * K;
    int row[KR];   // k * J + j: row k of virtual thread j; -1: none
    int e0[KR], len[KR];
    const int32_t* col;
    const V* val;
    double* sval;
    int32_t* scol;
    int width, slots;
};

template <typename V, int J, int K>
__device__ __forceinline__ void cg_load_rows(CgRows<V, J, K>& A, const CgGroup& g, int R, const int32_t* row_ptr,
                                             const int32_t* col, const V* val, unsigned char* smem, int smem_bytes)
{
    constexpr int KR = J * K;
    const unsigned halves = blockDim.x / kCgVirtual;
    A.slots = blockDim.x * KR;
    A.width = min(kCgRowSlots, smem_bytes / (A.slots * kCgEntryBytes));
    A.sval = reinterpret_cast<double*>(smem);
    A.scol = reinterpret_cast<int32_t*>(A.sval + (size_t)A.width * A.slots);
    A.col = col;
    A.val = val;
#pragma unroll
    for (int j = 0; j < KR; ++j) {
        const unsigned vb = (g.b * J + j % J) * halves + threadIdx.x / kCgVirtual;
        const int i = vb < g.vgrid ? (int)((j / J * g.vgrid + vb) * kCgVirtual + threadIdx.x % kCgVirtual) : R;
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
template <typename V, int J, int K, typename F>
__device__ __forceinline__ double cg_row_apply(const CgRows<V, J, K>& A, int j, double s, F&& x)
{
    const double* v = A.sval + j * blockDim.x + threadIdx.x;
    const int32_t* c = A.scol + j * blockDim.x + threadIdx.x;
    if (A.width == kCgRowSlots) {
        double xv[kCgRowSlots];
#pragma unroll
        for (int k = 0; k < kCgRowSlots; ++k) xv[k] = x(c[k * A.slots]);
#pragma unroll
        for (int k = 0; k < kCgRowSlots; ++k) s = fma(v[k * A.slots], xv[k], s);
    } else {
        for (int k = 0; k < A.width; ++k) s = fma(v[k * A.slots], x(c[k * A.slots]), s);
    }
    for (int k = A.width; k < A.len[j]; ++k) s = fma((double)__ldg(A.val + A.e0[j] + k), x(__ldg(A.col + A.e0[j] + k)), s);
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

template <typename V, int J, int K>
__device__ __forceinline__ void cg_iterate(CgGroup& g, const CgRows<V, J, K>& A, const double (&diag)[J * K],
                                           const double (&dinv)[J * K], double (&x)[J * K], double (&r)[J * K],
                                           double (&z)[J * K], double2* zp, CgScalars& c)
{
    constexpr int KR = J * K;
    double p[KR];
#pragma unroll
    for (int j = 0; j < KR; ++j) p[j] = 0.0;
    while (!c.done && !g.dead) {
        const double beta = c.iter == 0 ? 0.0 : c.rz / c.rz_prev;
        double q[KR], acc[1][J] = {}, sum[1], dots[2][J] = {}, sums[2];
#pragma unroll
        for (int j = 0; j < KR; ++j) {
            q[j] = 0.0;
            if (A.row[j] < 0) continue;
            const double pi = fma(beta, p[j], z[j]);
            const double s = cg_row_apply(A, j, __dmul_rn(diag[j], pi), [&](int c0) {
                const double2 n = zp[c0];  // by L1: a block's rows are neighbours
                return fma(beta, n.y, n.x);
            });
            p[j] = as_stored<V>(pi);
            q[j] = as_stored<V>(s);
            acc[0][j % J] = fma(pi, s, acc[0][j % J]);
        }
        group_sync_dots<1, J, false>(g, acc, sum);
        const double pq = sum[0];
        const double alpha = pq > 0.0 ? c.rz / pq : 0.0;
#pragma unroll
        for (int j = 0; j < KR; ++j) {
            if (A.row[j] < 0) continue;
            const double ri = fma(-alpha, q[j], r[j]);
            const double zi = __dmul_rn(ri, dinv[j]);
            x[j] = as_stored<V>(fma(alpha, p[j], x[j]));
            r[j] = as_stored<V>(ri);
            z[j] = as_stored<V>(zi);
            __stcg(zp + A.row[j], make_double2(z[j], p[j]));
            dots[0][j % J] = fma(ri, zi, dots[0][j % J]);
            dots[1][j % J] = fma(ri, ri, dots[1][j % J]);
        }
        group_sync_dots<2, J, true>(g, dots, sums);
        c.rz_prev = c.rz;
        c.rz = sums[0];
        c.rr = sums[1];
        c.iter += 1;
        if (c.rr <= c.thr2 || c.iter >= c.max_iter || !(pq > 0.0)) c.done = true;
    }
}

// FP64 CG from x (k_pcg_init + the k_pcg_spmv / k_pcg_update loop); zp: 2 R values.
template <int J, int K>
__device__ __forceinline__ void cg_solve64(CgGroup g, const PoissonView& P, const double* b, double* xg, double2* zp,
                                           PcgScalars* sc, double rtol, int max_iter, unsigned char* smem,
                                           int smem_bytes)
{
    constexpr int KR = J * K;
    CgRows<double, J, K> A;
    cg_load_rows(A, g, P.R, P.row_ptr, P.col, P.val, smem, smem_bytes);
    double x[KR], r[KR], z[KR], diag[KR], dinv[KR], acc[2][J] = {}, acc_b[1][J] = {}, sums[2], bb[1];
#pragma unroll
    for (int j = 0; j < KR; ++j) {
        x[j] = r[j] = z[j] = diag[j] = dinv[j] = 0.0;
        const int i = A.row[j];
        if (i < 0) continue;
        diag[j] = P.diag[i];
        dinv[j] = P.dinv ? P.dinv[i] : 1.0 / diag[j];
        x[j] = xg[i];
        const double bi = b[i];
        r[j] = bi - cg_row_apply(A, j, __dmul_rn(diag[j], x[j]), [&](int c0) { return __ldcg(xg + c0); });
        z[j] = __dmul_rn(r[j], dinv[j]);
        __stcg(zp + i, make_double2(z[j], 0.0));
        acc[0][j % J] = fma(r[j], z[j], acc[0][j % J]);
        acc[1][j % J] = fma(r[j], r[j], acc[1][j % J]);
        acc_b[0][j % J] = fma(bi, bi, acc_b[0][j % J]);
    }
    group_sync_dots<2, J, true>(g, acc, sums);
    group_sync_dots<1, J, false>(g, acc_b, bb);
    CgScalars c{};
    c.rz = sums[0];
    c.rz_prev = 1.0;
    c.rr = sums[1];
    c.thr2 = rtol * rtol * (bb[0] > 0.0 ? bb[0] : 1.0);
    c.max_iter = max_iter;
    c.done = c.rr <= c.thr2 || max_iter <= 0;
    cg_iterate<double, J, K>(g, A, diag, dinv, x, r, z, zp, c);
#pragma unroll
    for (int j = 0; j < KR; ++j)
        if (A.row[j] >= 0) xg[A.row[j]] = x[j];
    if (g.b == 0 && threadIdx.x == 0) {
        sc->rz = c.rz;
        sc->rz_prev = c.rz_prev;
        sc->rr = c.rr;
        sc->bb = bb[0];
        sc->thr2 = c.thr2;
        sc->iter = c.iter;
        sc->done = g.dead ? -1 : 1;
    }
}

// The precision form's solve: FP32 CG for the correction inside FP64 refinement (the loop of
// run_pcg_mixed in capi.cu), all passes in this call.  sc: rr, bb, iter (inner iterations in all)
// and outer (passes) out.
template <int J, int K>
__device__ __forceinline__ void cg_solve_mixed(CgGroup& g, const PoissonView& P, const double* b, double* xg,
                                               double2* zp, PcgScalars* sc, double rtol, int max_iter,
                                               unsigned char* smem, int smem_bytes)
{
    constexpr int KR = J * K;
    CgRows<float, J, K> A;
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
        double e[KR], r[KR], z[KR], acc[2][J] = {}, res[2][J] = {}, sums[2];
#pragma unroll
        for (int j = 0; j < KR; ++j) {
            e[j] = r[j] = z[j] = 0.0;
            const int i = A.row[j];
            if (i < 0) continue;
            // the FP64 matrix's values are read: two to four of these against an iteration each time
            double s = __dmul_rn(P.diag[i], x[j]);
            const double* val = P.val + A.e0[j];
            const int32_t* col = P.col + A.e0[j];
#pragma unroll 4
            for (int k = 0; k < A.len[j]; ++k) s = fma(__ldg(val + k), __ldcg(xg + __ldg(col + k)), s);
            const double bi = b[i], ri = bi - s;
            res[0][j % J] = fma(ri, ri, res[0][j % J]);
            res[1][j % J] = fma(bi, bi, res[1][j % J]);
            // the start of A e = r from e = 0
            r[j] = as_stored<float>(ri);
            const double zf = __dmul_rn(r[j], dinv[j]);
            z[j] = as_stored<float>(zf);
            __stcg(zp + i, make_double2(z[j], 0.0));
            acc[0][j % J] = fma(r[j], zf, acc[0][j % J]);
            acc[1][j % J] = fma(r[j], r[j], acc[1][j % J]);
        }
        group_sync_dots<2, J, true>(g, res, norm);
        const double bb = norm[1] > 0.0 ? norm[1] : 1.0;
        if (g.dead || norm[0] <= rtol * rtol * bb || iters >= max_iter || outer == kMaxRefinePasses) break;
        group_sync_dots<2, J, false>(g, acc, sums);
        // to the tolerance this pass needs
        const double rt = inner_rtol(norm[0], bb, rtol);
        CgScalars c{};
        c.rz = sums[0];
        c.rz_prev = 1.0;
        c.rr = sums[1];
        c.thr2 = rt * rt * (sums[1] > 0.0 ? sums[1] : 1.0);
        c.max_iter = max(1, max_iter - iters);
        c.done = c.rr <= c.thr2;
        cg_iterate<float, J, K>(g, A, diag, dinv, e, r, z, zp, c);
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
// grids: blocks of 256 threads of the launched form of each system (CgGroup::vgrid).
// blocks_of: blocks of each group.
CgPlan cg_plan(const int* rows, const int* grids, int n, int nsm, int* blocks_of);

// The runtime refused a cooperative launch: the launched form can run instead.
inline bool cg_refused(cudaError_t e)
{
    return e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported;
}

// Cooperative, since a group's blocks wait on one another and all have to be resident; a refusal is the
// returned value only.
inline cudaError_t cg_launch(const void* kernel, int blocks, int threads, void** args, size_t smem, cudaStream_t st)
{
    const cudaError_t e = cudaLaunchCooperativeKernel(kernel, dim3(blocks), dim3(threads), args, smem, st);
    if (cg_refused(e)) cudaGetLastError();
    return e;
}

// One system: queues the solve on st.  zp: 2 R values; slots: kCgSlotBytes; grid: as for cg_plan; results
// in sc (done < 0: a barrier wait ran out).
cudaError_t launch_cg64(const CgPlan& plan, int grid, const PoissonView& A, const double* b, double* x, double* zp,
                        PcgScalars* sc, double* slots, double rtol, int max_iter, cudaStream_t st);
cudaError_t launch_cg_mixed(const CgPlan& plan, int grid, const PoissonView& A, const double* b, double* x, double* zp,
                            PcgScalars* sc, double* slots, double rtol, int max_iter, cudaStream_t st);

// f(J, K) as integral constants for the plan's rows per thread.
template <typename F>
auto cg_dispatch(const CgPlan& p, F&& f)
{
    using std::integral_constant;
    if (p.rounds == 2) {
        if (p.virt == 1) return f(integral_constant<int, 1>{}, integral_constant<int, 2>{});
        return f(integral_constant<int, 2>{}, integral_constant<int, 2>{});
    }
    if (p.rounds == 3) return f(integral_constant<int, 1>{}, integral_constant<int, 3>{});
    if (p.rounds == 4) return f(integral_constant<int, 1>{}, integral_constant<int, 4>{});
    if (p.virt == 1) return f(integral_constant<int, 1>{}, integral_constant<int, 1>{});
    if (p.virt == 2) return f(integral_constant<int, 2>{}, integral_constant<int, 1>{});
    if (p.virt == 3) return f(integral_constant<int, 3>{}, integral_constant<int, 1>{});
    return f(integral_constant<int, 4>{}, integral_constant<int, 1>{});
}

}  // namespace scdat
