// push_f64.cu -- the plain FP64 particle step: one thread per particle runs
// CrossTetrahedron::integrateTrajectory (PICParticleAlgorithms.cpp:536-740) with the
// adaptive sub-step (:750-801), Boris with B = 0 (:803-851), relocation (:853-891) and the
// per-sub-step trajectory deposit (:371-433), then the runtime boundary events
// (PICCycle.cpp:1221-1379) and, when enabled, the elastic background MCC.
//
// Charge goes into per-species 128-bit fixed-point node accumulators, so the deposit is exact and
// independent of thread order.  The nodal E of each tet's 4 nodes is kept per tet (refreshed after
// every field solve), so the gather is one load beside the tet's geometry.  Sub-steps run in passes
// to keep warps converged, and pass 1 walks from a queue and ends the rare cases in pass 2, as in
// push_mixed.cu.
#include "push.cuh"
#include "segment_cloud.h"

namespace scdat {

constexpr int kPushWarpsD = 8, kPushBlocksD = 2;  // pass 1: warps of a block, blocks per SM

// The inverse Jacobian (row-major) and origin of a tet's record.
struct TetGeom {
    double j[9], o[3];
};

__device__ __forceinline__ TetGeom load_geom(const MeshView& M, int t)
{
    const double2* g2 = reinterpret_cast<const double2*>(M.geom + 16 * (int64_t)t);
    const double2 a = __ldg(g2), b = __ldg(g2 + 1), c = __ldg(g2 + 2), d = __ldg(g2 + 3), e = __ldg(g2 + 4),
                  f = __ldg(g2 + 5);
    return TetGeom{{a.x, a.y, b.x, b.y, c.x, c.y, d.x, d.y, e.x}, {e.y, f.x, f.y}};
}

// bary64 from a record already in registers.  The rounding is spelled out: left to the compiler, two
// uses contracted differently, and a step taken up again in pass 3 could end 1 ulp from one that ran on.
__device__ __forceinline__ bool baryg(const TetGeom& g, double px, double py, double pz, double lam[4])
{
    const double dx = px - g.o[0], dy = py - g.o[1], dz = pz - g.o[2];
    lam[1] = fma(g.j[2], dz, fma(g.j[1], dy, __dmul_rn(g.j[0], dx)));
    lam[2] = fma(g.j[5], dz, fma(g.j[4], dy, __dmul_rn(g.j[3], dx)));
    lam[3] = fma(g.j[8], dz, fma(g.j[7], dy, __dmul_rn(g.j[6], dx)));
    lam[0] = 1.0 - lam[1] - lam[2] - lam[3];
    return bary_inside(lam);
}

// ChargeDepositor::depositChargeAlongTrajectory into the post-move tet t, whose record is g
// (PICParticleAlgorithms.cpp:371-433); each sample point counts only when it lies in t.
__device__ __forceinline__ void deposit_traj(const MeshView& M, const SpeciesDev& S, const PushParams& pp, int t,
                                             const TetGeom& g, double sx, double sy, double sz, double ex, double ey,
                                             double ez, ChargeAcc A)
{
    TwoDouble sum[4] = {};  // the sample points' contributions, exact until the 128-bit node words take them
    bool any = false;
    const double tx = ex - sx, ty = ey - sy, tz = ez - sz;
    const double qw = S.q * S.w;
    const bool tiny = sqrt(tx * tx + ty * ty + tz * tz) < 1e-15;
    if (tiny || pp.dep_kernel == 0) {  // a point: the start of a tiny move, NearestPoint's end
        double lam[4];
        any = tiny ? baryg(g, sx, sy, sz, lam) : baryg(g, ex, ey, ez, lam);
#pragma unroll
        for (int i = 0; i < 4; ++i) sum[i].hi = seg_mul(qw, lam[i]);
    } else {
        // barycentrics are affine along the segment: lam(s + tau*tr) = lam_s + tau*dlam
        double ls[4], dl[4];
        baryg(g, sx, sy, sz, ls);
        dl[1] = g.j[0] * tx + g.j[1] * ty + g.j[2] * tz;
        dl[2] = g.j[3] * tx + g.j[4] * ty + g.j[5] * tz;
        dl[3] = g.j[6] * tx + g.j[7] * ty + g.j[8] * tz;
        dl[0] = -dl[1] - dl[2] - dl[3];
        const int nseg = pp.nseg;
        if (pp.dep_kernel == 2) {  // QuadratureGauss3
            const double gn[3] = {-0.7745966692414834, 0.0, 0.7745966692414834};
            const double gw[3] = {5.0 / 18.0, 8.0 / 18.0, 5.0 / 18.0};
            for (int sg = 0; sg < nseg; ++sg) {
                double t0 = (double)sg / (double)nseg, t1 = (double)(sg + 1) / (double)nseg;
                double tc = 0.5 * (t0 + t1), th = 0.5 * (t1 - t0);
                for (int q = 0; q < 3; ++q) {
                    double tau = tc + th * gn[q];
                    double l[4] = {ls[0] + tau * dl[0], ls[1] + tau * dl[1], ls[2] + tau * dl[2], ls[3] + tau * dl[3]};
                    if (bary_inside(l)) {
                        const double cw = (S.q * gw[q] / (double)nseg) * S.w;
#pragma unroll
                        for (int i = 0; i < 4; ++i) seg_add(sum[i], seg_mul(cw, l[i]));
                        any = true;
                    }
                }
            }
        } else {
            // LinearSegmentCloud: the points inside the tet, whose sum is in closed form
            const SegPoints p = seg_points(ls, dl, nseg, kBaryEps);
            any = p.first <= p.last;
#pragma unroll
            for (int i = 0; i < 4; ++i) sum[i] = seg_sum(ls[i], dl[i], p, nseg, S.cw_seg);
        }
    }
    if (!any) return;
    const int4 tn = rec_nodes(M, t);
    fx_red(A, tn.x, sum[0].hi * pp.inv_uq, sum[0].lo * pp.inv_uq);
    fx_red(A, tn.y, sum[1].hi * pp.inv_uq, sum[1].lo * pp.inv_uq);
    fx_red(A, tn.z, sum[2].hi * pp.inv_uq, sum[2].lo * pp.inv_uq);
    fx_red(A, tn.w, sum[3].hi * pp.inv_uq, sum[3].lo * pp.inv_uq);
}

struct FlightD {
    double px, py, pz, vx, vy, vz;
    double rem, vstart;
    int cur, it;
};

// The gathered field of a sub-step at barycentrics lam (zero outside the tet), its length in time
// (CrossTetrahedron::adaptiveTimeStep with |B| = 0), and the velocity after its two half kicks.
__device__ __forceinline__ double kick_d(const MeshView& M, const SpeciesDev& S, const PushParams& pp,
                                         const double lam[4], bool in, FlightD& f)
{
    const double qm = S.qm;
    double Ex = 0.0, Ey = 0.0, Ez = 0.0;
    if (in) {
        const double2* e2 = reinterpret_cast<const double2*>(M.erec + 12 * (int64_t)f.cur);
        const double2 a = __ldg(e2), b = __ldg(e2 + 1), c = __ldg(e2 + 2), d = __ldg(e2 + 3), g = __ldg(e2 + 4),
                      h = __ldg(e2 + 5);
        const double e[12] = {a.x, a.y, b.x, b.y, c.x, c.y, d.x, d.y, g.x, g.y, h.x, h.y};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            Ex = Ex + e[3 * q] * lam[q];
            Ey = Ey + e[3 * q + 1] * lam[q];
            Ez = Ez + e[3 * q + 2] * lam[q];
        }
    }
    double adt = f.rem;
    const double Em = sqrt(Ex * Ex + Ey * Ey + Ez * Ez);
    if (Em > 1e-10) {
        const double acc = Em * fabs(qm);
        if (acc > 1e-10 && f.vstart > 1.0) adt = fmin(adt, 0.1 * f.vstart / acc);
    }
    adt = fmax(adt, f.rem * pp.floor_ratio);
    adt = fmin(adt, f.rem);
    if (fabs(qm) > 1e-20) {
        const double h = qm * (0.5 * adt);
        f.vx = f.vx + Ex * h; f.vy = f.vy + Ey * h; f.vz = f.vz + Ez * h;
        f.vx = f.vx + Ex * h; f.vy = f.vy + Ey * h; f.vz = f.vz + Ez * h;
    }
    return adt;
}

// Deposit of a sub-step that stayed in its tet (see deposit_in_f in push_mixed.cu).
__device__ __forceinline__ void deposit_in_d(const MeshView& M, const SpeciesDev& S, const PushParams& pp, int t,
                                             const double lam[4], const double le[4], double tx, double ty, double tz,
                                             ChargeAcc A)
{
    const double qw = S.q * S.w;
    const bool tiny = sqrt(tx * tx + ty * ty + tz * tz) < 1e-15;
    const int4 tn = rec_nodes(M, t);
    const int nd[4] = {tn.x, tn.y, tn.z, tn.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const double lk = tiny ? lam[q] : (pp.dep_kernel == 0 ? le[q] : 0.5 * (lam[q] + le[q]));
        fx_red(A, nd[q], (qw * lk) * pp.inv_uq);
    }
}

// Run sub-steps until the step's time is used up, the particle is lost, or `cap` sub-steps
// ran in this call.
__device__ __forceinline__ int advance_d(const MeshView& M, const SpeciesDev& S, const PushParams& pp, FlightD& f,
                                         int cap, ChargeAcc A,
                                         unsigned& nsub)
{
    TetGeom g = load_geom(M, f.cur);
    double lam[4];
    bool in = baryg(g, f.px, f.py, f.pz, lam);  // reused as the next gather's weights
    int k = 0;
    while (f.rem > kMinTimeStep && f.it < kMaxSubsteps) {
        if (k == cap) return kCapped;
        ++k;
        ++f.it;
        const double sx = f.px, sy = f.py, sz = f.pz;
        const double adt = kick_d(M, S, pp, lam, in, f);
        f.px = fma(f.vx, adt, sx);
        f.py = fma(f.vy, adt, sy);
        f.pz = fma(f.vz, adt, sz);
        double le[4];
        if (baryg(g, f.px, f.py, f.pz, le)) {
            if (pp.deposit) {
                if (in)
                    deposit_in_d(M, S, pp, f.cur, lam, le, f.px - sx, f.py - sy, f.pz - sz, A);
                else
                    deposit_traj(M, S, pp, f.cur, g, sx, sy, sz, f.px, f.py, f.pz, A);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) lam[q] = le[q];
            in = true;
        } else {
            const int nt = locate(M, f.px, f.py, f.pz, f.cur);
            if (nt < 0) return kLost;
            f.cur = nt;
            g = load_geom(M, nt);
            if (pp.deposit) deposit_traj(M, S, pp, nt, g, sx, sy, sz, f.px, f.py, f.pz, A);
            in = baryg(g, f.px, f.py, f.pz, lam);
        }
        f.rem -= adt;
        ++nsub;
    }
    return f.it >= kMaxSubsteps ? kLost : kDone;
}

// The end of a particle's step in tet `tet` (< 0: inactive), with the fused MCC when COLLIDE.
template <bool COLLIDE>
__device__ __forceinline__ void finish_in_d(const ParticleStore& P, const SpeciesDev& S, const PushParams& pp,
                                            int64_t i, FlightD& f, int tet, double ke, PushStats& c)
{
    c.ke += ke;  // updateStatistics counts every stored particle (PICCycle.cpp:941-966)
    if (tet >= 0) {
        c.ev |= kEvActive;
        if (S.mcc_mode == 2) c.v2 = fmaxf(c.v2, (float)(f.vx * f.vx + f.vy * f.vy + f.vz * f.vz));  // the null-collision speed bound
        if (COLLIDE && pp.do_mcc && S.mcc_enabled && mcc_elastic(S, pp, P.id[i], f.vx, f.vy, f.vz)) c.ev |= kEvHit;
    }
    P.x[i] = f.px; P.y[i] = f.py; P.z[i] = f.pz;
    P.vx[i] = f.vx; P.vy[i] = f.vy; P.vz[i] = f.vz;
    P.tet[i] = tet;
}

__device__ __forceinline__ void finish_d(const MeshView& M, const ParticleStore& P, const SpeciesDev& S,
                                         const PushParams& pp, LedgerDev* L, int64_t i, FlightD& f, int st,
                                         PushStats& c)
{
    const double ke = 0.5 * S.m * (f.vx * f.vx + f.vy * f.vy + f.vz * f.vz);
    int tet_out = f.cur;
    if (st == kLost) {
        c.ev |= kEvLost;
        // lost before the sub-step cap: no tet holds the position
        tet_out = resolve_lost(M, S, pp, L, f.px, f.py, f.pz, ke, f.cur, f.it < kMaxSubsteps);
    }
    finish_in_d<true>(P, S, pp, i, f, tet_out, ke, c);
}

__device__ __forceinline__ void defer_store_d(const ParticleStore& P, const DeferList& D, unsigned slot, int64_t i,
                                              const FlightD& f)
{
    D.idx[slot] = (uint32_t)i;
    D.it[slot] = f.it;
    D.rem[slot] = f.rem;
    D.vstart[slot] = f.vstart;
    P.x[i] = f.px; P.y[i] = f.py; P.z[i] = f.pz;
    P.vx[i] = f.vx; P.vy[i] = f.vy; P.vz[i] = f.vz;
    P.tet[i] = f.cur;
}

// A warp's particles that left their tet in pass 1 and wait for their walk (see push_mixed.cu).
struct WalkQueueD {
    double sx[kWalkQueue], sy[kWalkQueue], sz[kWalkQueue], vx[kWalkQueue], vy[kWalkQueue], vz[kWalkQueue];
    double adt[kWalkQueue], vstart[kWalkQueue];
    uint32_t i[kWalkQueue];
    int cur[kWalkQueue];
};

__device__ __forceinline__ WalkQueueD& walk_queue_d()
{
    __shared__ WalkQueueD q[kPushWarpsD];
    return q[threadIdx.x >> 5];
}

// End of a particle's pass-1 sub-step (see end_first in push_mixed.cu).
template <bool COLLIDE>
__device__ __forceinline__ void end_first_d(const ParticleStore& P, const SpeciesDev& S, const PushParams& pp,
                                            const DeferList& D, LedgerDev* L, int64_t i, FlightD& f, int st,
                                            PushStats& c)
{
    double ke = 0.0;
    if (st == kDone) {
        const double v2 = f.vx * f.vx + f.vy * f.vy + f.vz * f.vz;
        ke = 0.5 * S.m * v2;
        if (!COLLIDE && pp.do_mcc && S.mcc_enabled && mcc_candidate(S, pp, P.id[i], v2)) st = kFinish;
    }
    const bool more = st > kDone;
    const unsigned slot = warp_append(more, D.count);
    if (more) {
        f.it = st == kLost ? kItLost : (st == kFinish ? kItFinish : f.it);
        if (slot < D.cap)
            defer_store_d(P, D, slot, i, f);
        else
            atomicOr(&L->flags, (unsigned long long)kFlagDeferOverflow);  // the step fails with this flag
    } else if (st == kDone) {
        finish_in_d<COLLIDE>(P, S, pp, i, f, f.cur, ke, c);
    }
    warp_chunk_end(c);
}

// Walks m (up to 32) particles of the warp's queue from position `first` on: locate()'s walk from the
// tet they left and the deposit in the tet they reach.  Points outside the domain are lost; those
// the walk does not settle (a boundary face, a long walk, the tolerance band of several tets) run
// again in pass 2, in the reference's search order.
template <bool COLLIDE>
__device__ __forceinline__ void walk_queued_d(const MeshView& M, const ParticleStore& P, const SpeciesDev& S,
                                              const PushParams& pp, const DeferList& D, ChargeAcc A, LedgerDev* L,
                                              int first, int m, PushStats& c)
{
    const int lane = threadIdx.x & 31;
    const WalkQueueD& Q = walk_queue_d();
    const int e = first + lane;
    int st = -1;
    int64_t i = 0;
    FlightD f;
    __syncwarp();
    if (lane < m) {
        i = Q.i[e];
        const double adt = Q.adt[e];
        f.vstart = Q.vstart[e];
        f.px = fma(Q.vx[e], adt, Q.sx[e]);
        f.py = fma(Q.vy[e], adt, Q.sy[e]);
        f.pz = fma(Q.vz[e], adt, Q.sz[e]);
        f.cur = Q.cur[e];
        f.it = 1;
        f.rem = pp.dt - adt;
        st = kLost;
        if (!outside_grid(M, f.px, f.py, f.pz)) {
            st = kRedo;
            int t = f.cur;
            TetGeom g;
            for (int k = 0; k < kWalkSteps; ++k) {
                double lam[4];
                g = load_geom(M, t);
                const bool inside = baryg(g, f.px, f.py, f.pz, lam);
                const double mn = fmin(fmin(lam[0], lam[1]), fmin(lam[2], lam[3]));
                if (!(mn == mn)) break;
                if (inside) {
                    if (mn >= 1e-6) st = kDone;
                    break;
                }
                int fc = 0;
                double lm = lam[0];
                if (lam[1] < lm) { lm = lam[1]; fc = 1; }
                if (lam[2] < lm) { lm = lam[2]; fc = 2; }
                if (lam[3] < lm) fc = 3;
                const int nt = __ldg(reinterpret_cast<const int*>(M.geom + 16 * (int64_t)t + 12) + fc);
                if (nt < 0) break;
                t = nt;
            }
            if (st == kDone) {
                if (pp.deposit) deposit_traj(M, S, pp, t, g, Q.sx[e], Q.sy[e], Q.sz[e], f.px, f.py, f.pz, A);
                f.cur = t;
                ++c.nsub;
                if (f.rem > kMinTimeStep) st = kCapped;
            }
        }
        f.vx = Q.vx[e]; f.vy = Q.vy[e]; f.vz = Q.vz[e];
        if (st == kRedo) {  // the state of the step's start is still in the store
            f.px = P.x[i]; f.py = P.y[i]; f.pz = P.z[i];
            f.vx = P.vx[i]; f.vy = P.vy[i]; f.vz = P.vz[i];
            f.rem = pp.dt;
            f.it = 0;
        }
    }
    end_first_d<COLLIDE>(P, S, pp, D, L, i, f, st, c);
}

// Pass 1 for the 32 particles [base, base + 32) of one warp: one sub-step, the leavers queued.
template <bool COLLIDE>
__device__ __forceinline__ void push1_warp_d(const MeshView& M, const ParticleStore& P, const SpeciesDev& S,
                                             const PushParams& pp, const DeferList& D, ChargeAcc A, LedgerDev* L,
                                             int64_t base, int64_t n, int& queued, PushStats& c)
{
    static_assert(kCap1 == 1, "pass 1 runs one sub-step");
    const int lane = threadIdx.x & 31;
    const int64_t i = base + lane;
    int st = -1;
    bool leaves = false;
    FlightD f;
    double adt = 0.0;
    if (i < n) {
        f.cur = P.tet[i];
        f.vx = P.vx[i]; f.vy = P.vy[i]; f.vz = P.vz[i];
        if (f.cur <= kTetAbsorbed) {
            // updateStatistics sums every particle the container still holds (PICCycle.cpp:941-966)
            c.ke += 0.5 * S.m * (f.vx * f.vx + f.vy * f.vy + f.vz * f.vz);
        } else {
            f.px = P.x[i]; f.py = P.y[i]; f.pz = P.z[i];
            f.vstart = sqrt(f.vx * f.vx + f.vy * f.vy + f.vz * f.vz);
            f.rem = pp.dt;
            f.it = 0;
            st = kRedo;  // no hint, or a hint that does not hold the point: located by pass 2
            TetGeom g;
            double lam[4];
            bool in = false;
            if (f.cur >= 0) {
                g = load_geom(M, f.cur);
                in = baryg(g, f.px, f.py, f.pz, lam);
            }
            if (in) {
                st = kDone;
                if (f.rem > kMinTimeStep) {
                    const double sx = f.px, sy = f.py, sz = f.pz;
                    adt = kick_d(M, S, pp, lam, true, f);
                    f.px = fma(f.vx, adt, sx);
                    f.py = fma(f.vy, adt, sy);
                    f.pz = fma(f.vz, adt, sz);
                    double le[4];
                    if (baryg(g, f.px, f.py, f.pz, le)) {
                        if (pp.deposit)
                            deposit_in_d(M, S, pp, f.cur, lam, le, f.px - sx, f.py - sy, f.pz - sz, A);
                        f.rem -= adt;
                        f.it = 1;
                        ++c.nsub;
                        if (f.rem > kMinTimeStep) st = kCapped;
                    } else {
                        leaves = true;
                        f.px = sx; f.py = sy; f.pz = sz;
                    }
                }
            }
        }
    }
    const unsigned m = __ballot_sync(0xffffffffu, leaves);
    if (leaves) {
        const int e = queued + __popc(m & ((1u << lane) - 1u));
        WalkQueueD& Q = walk_queue_d();
        Q.i[e] = (uint32_t)i;
        Q.cur[e] = f.cur;
        Q.sx[e] = f.px; Q.sy[e] = f.py; Q.sz[e] = f.pz;
        Q.vx[e] = f.vx; Q.vy[e] = f.vy; Q.vz[e] = f.vz;
        Q.adt[e] = adt;
        Q.vstart[e] = f.vstart;
        st = -1;
    }
    queued += __popc(m);
    end_first_d<COLLIDE>(P, S, pp, D, L, i, f, st, c);
}

// Pass 1: every stored particle, one sub-step, in runs of chunks (see k_push_mixed).  Bound by the
// latency of the records' loads at the 16 warps per SM its registers leave.  Two species of 3.5 M
// particles at 48^3 cells, both launches: 2.24 ms with locate and a sample-by-sample deposit out of
// line in the chunk's flow (14 of 32 threads active), 1.10 ms now; 3 blocks per SM (80 registers,
// 346 bytes of spills) 1.25, 5 blocks of 4 warps (96 registers, 172 bytes) 1.19.
template <bool COLLIDE>
__global__ void __launch_bounds__(32 * kPushWarpsD, kPushBlocksD)
    k_push_f64(const __grid_constant__ MeshView M, const __grid_constant__ ParticleStore P,
               const __grid_constant__ SpeciesDev S, const __grid_constant__ PushParams pp, DeferList D, ChargeAcc A,
               LedgerDev* L, unsigned long long* ke_acc, unsigned* ctr)
{
    const int64_t n = *P.count;
    PushStats c{0.0, 0u, 0u};
    const int64_t run = 32 * run_chunks(n, (int64_t)gridDim.x * (blockDim.x >> 5));
    warp_stats_begin();
    int64_t base = 0, end = 0;
    int queued = 0;
    for (bool left = true;;) {
        if (queued >= 32 || (!left && queued > 0)) {
            const int m = min(queued, 32);
            queued -= m;
            walk_queued_d<COLLIDE>(M, P, S, pp, D, A, L, queued, m, c);
        } else if (!left) {
            break;
        } else if (base < end) {
            push1_warp_d<COLLIDE>(M, P, S, pp, D, A, L, base, n, queued, c);
            base += 32;
        } else {
            base = (int64_t)next_chunk(ctr) * run;
            end = min(base + run, n);
            left = base < n;
        }
    }
    warp_stats_flush(L, ke_acc, S.vmax);
}

// Passes 2 and 3 over a deferred list (see k_push_mixed_more).
__global__ void __launch_bounds__(256) k_push_f64_more(const __grid_constant__ MeshView M, ParticleStore P,
    const __grid_constant__ SpeciesDev S, const __grid_constant__ PushParams pp,
                                                       DeferList Din, DeferList Dout, int cap, ChargeAcc A, LedgerDev* L,
                                                       unsigned long long* ke_acc, unsigned* ctr)
{
    const int64_t n = (int64_t)min(*Din.count, Din.cap);
    if (n == 0) return;  // 3 us; every warp's first atomic on the work counter alone takes 9
    PushStats c{0.0, 0u, 0u};
    const int lane = threadIdx.x & 31;
    const bool chain = Dout.count != nullptr;
    int64_t base, end;
    const bool once = list_share(n, base, end);
    if (once && base >= n) return;
    if (once) cap = 0x7fffffff;
    warp_stats_begin();
    for (;;) {
        if (!once) {
            base = (int64_t)next_chunk(ctr) * 32;
            end = n;
            if (base >= n) break;
        }
        const int64_t e = base + lane;
        int st = -1;
        FlightD f;
        int64_t i = 0;
        if (e < end) {
            i = Din.idx[e];
            f.cur = P.tet[i];
            f.px = P.x[i]; f.py = P.y[i]; f.pz = P.z[i];
            f.vx = P.vx[i]; f.vy = P.vy[i]; f.vz = P.vz[i];
            f.it = Din.it[e];
            f.rem = Din.rem[e];
            f.vstart = Din.vstart[e];
            const bool ends = f.it < 0;  // kItLost, kItFinish: only the end of the step is left
            st = f.it == kItLost ? kLost : kDone;
            if (f.it == 0) {
                // the whole step: pass 1 did not find it in its hint, or did not settle its walk
                f.cur = locate(M, f.px, f.py, f.pz, f.cur);
                if (f.cur < 0) {
                    f.cur = 0;  // result.final_element stays 0 (PICParticleAlgorithms.cpp:543,577)
                    st = kLost;
                }
            }
            if (!ends && st != kLost) st = advance_d(M, S, pp, f, chain ? cap : 0x7fffffff, A, c.nsub);
        }
        unsigned slot = chain ? warp_append(st == kCapped, Dout.count) : 0xffffffffu;
        if (st == kCapped && chain && slot < Dout.cap) {
            defer_store_d(P, Dout, slot, i, f);
        } else if (st >= 0) {
            if (st == kCapped) st = advance_d(M, S, pp, f, 0x7fffffff, A, c.nsub);
            finish_d(M, P, S, pp, L, i, f, st, c);
        }
        warp_chunk_end(c);
        if (once) break;
    }
    warp_stats_flush(L, ke_acc, S.vmax);
}

// Standalone MCC pass (executeBackgroundMccStep, CollisionPicAdapter.cpp:338-434).
__global__ void k_mcc_f64(ParticleStore P, SpeciesDev S, PushParams pp, LedgerDev* L)
{
    const int64_t n = *P.count;
    unsigned long long nhit = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        if (P.tet[i] <= kTetAbsorbed) continue;
        double vx = P.vx[i], vy = P.vy[i], vz = P.vz[i];
        if (mcc_elastic(S, pp, P.id[i], vx, vy, vz)) {
            P.vx[i] = vx; P.vy[i] = vy; P.vz[i] = vz;
            ++nhit;
        }
    }
    if (nhit) atomicAdd(&L->mcc_hits, nhit);
}

// Per-tet copy of the nodal E of its 4 nodes.
__global__ void k_refresh_erec(int64_t T, const int4* __restrict__ tet, const double* __restrict__ E, double* erec)
{
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < T; t += (int64_t)gridDim.x * blockDim.x) {
        int4 tn = tet[t];
        int nd[4] = {tn.x, tn.y, tn.z, tn.w};
        double* r = erec + 12 * t;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            r[3 * q] = E[3 * (int64_t)nd[q]];
            r[3 * q + 1] = E[3 * (int64_t)nd[q] + 1];
            r[3 * q + 2] = E[3 * (int64_t)nd[q] + 2];
        }
    }
}

void launch_push_f64(const MeshView& M, const ParticleStore& P, const SpeciesDev& S, const PushParams& pp,
                     const DeferList& D1, const DeferList& D2, ChargeAcc A, LedgerDev* L, unsigned long long* ke_acc,
                     unsigned* ctr, int grid, cudaStream_t st)
{
    auto first = pp.do_mcc && S.mcc_enabled && S.mcc_mode != 2 ? k_push_f64<true> : k_push_f64<false>;
    first<<<grid * (8 / kPushWarpsD), 32 * kPushWarpsD, 0, st>>>(M, P, S, pp, D1, A, L, ke_acc, ctr);
    grid = std::min(grid, 148 * 2);  // what is resident at once
    k_push_f64_more<<<grid, 256, 0, st>>>(M, P, S, pp, D1, D2, kCap2, A, L, ke_acc, ctr + 1);
    DeferList none{};
    k_push_f64_more<<<grid, 256, 0, st>>>(M, P, S, pp, D2, none, 0, A, L, ke_acc, ctr + 2);
}

void launch_mcc_f64(const ParticleStore& P, const SpeciesDev& S, const PushParams& pp, LedgerDev* L, int grid,
                    cudaStream_t st)
{
    k_mcc_f64<<<grid, 256, 0, st>>>(P, S, pp, L);
}

void launch_refresh_erec(int64_t T, const int4* tet, const double* E, double* erec, cudaStream_t st)
{
    k_refresh_erec<<<148 * 8, 256, 0, st>>>(T, tet, E, erec);
}

}  // namespace scdat
