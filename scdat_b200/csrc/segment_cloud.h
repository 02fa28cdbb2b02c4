// segment_cloud.h -- the sample points of LinearSegmentCloud (PICParticleAlgorithms.cpp:371-433) that lie in a
// tet, in closed form (host and device; the FP64 push).  Barycentrics are affine along the segment,
// l_i(tau) = ls[i] + tau * dl[i], so the points tau_k = (k + 1/2) / nseg inside are those of one interval of k.
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define SCDAT_SEG __host__ __device__ __forceinline__
#else
#define SCDAT_SEG inline
#endif

namespace scdat {

// Points first to last; none when last < first.
struct SegPoints {
    int first, last;
};

SCDAT_SEG bool seg_inside(const double* ls, const double* dl, int nseg, double eps, int k)
{
    const double tau = ((double)k + 0.5) / (double)nseg;
    bool ok = true;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const double l = fma(tau, dl[i], ls[i]);
        ok = ok && l >= -eps && l <= 1.0 + eps;
    }
    return ok;
}

// The interval's ends come from the faces' crossings and are settled by the containment test of the points
// next to them, so that they are the points a loop over all of them would take.  A crossing is off by
// about 1e-16 / |dl| in tau, less than a point for nseg <= 128 and |dl| over 1e-13; below kSegMinStep the
// rounding of l_i decides at many points, and the tests alone do: each l_i is monotone in k, so trimming
// from both ends finds the interval.
constexpr double kSegMinStep = 1e-12;

SCDAT_SEG SegPoints seg_points(const double* ls, const double* dl, int nseg, double eps)
{
    double lo = 0.0, hi = 1.0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (fabs(dl[i]) < kSegMinStep) continue;
        const double inv = 1.0 / dl[i];
        const double a = (-eps - ls[i]) * inv, b = (1.0 + eps - ls[i]) * inv;
        lo = fmax(lo, fmin(a, b));
        hi = fmin(hi, fmax(a, b));
    }
    const double n = (double)nseg;
    int a = (int)fmin(fmax(ceil(lo * n - 0.5), 0.0), n);
    int b = (int)fmax(fmin(floor(hi * n - 0.5), n - 1.0), -1.0);
    if (a > 0 && seg_inside(ls, dl, nseg, eps, a - 1)) --a;
    if (b < nseg - 1 && seg_inside(ls, dl, nseg, eps, b + 1)) ++b;
    while (a <= b && !seg_inside(ls, dl, nseg, eps, a)) ++a;
    while (b >= a && !seg_inside(ls, dl, nseg, eps, b)) --b;
    return SegPoints{a, b};
}

// A value and what its rounding lost.
struct TwoDouble {
    double hi, lo;
};

SCDAT_SEG double seg_mul(double a, double b)  // rounded: not contracted with what it is added to
{
#ifdef __CUDA_ARCH__
    return __dmul_rn(a, b);
#else
    return a * b;
#endif
}

// a + v: the sum of FP64 terms without their rounding errors' loss
SCDAT_SEG void seg_add(TwoDouble& a, double v)
{
    const double s = a.hi + v, z = s - a.hi;
    a.lo += (a.hi - (s - z)) + (v - z);
    a.hi = s;
}

// The sum of c * l(tau_k) over n points from `first`, c * (n ls + m / nseg dl) with m the sum of k + 1/2.  The
// sample points' contributions used to be rounded one by one and added exactly; this carries what each
// product and sum rounds away, so that it is no further from the exact sum.
SCDAT_SEG TwoDouble seg_sum(double ls, double dl, SegPoints p, int nseg, double c)
{
    const double n = (double)(p.last - p.first + 1), m = 0.5 * n * (double)(p.first + p.last + 1);  // exact
    const double inv = 1.0 / (double)nseg, t = seg_mul(m, inv), tl = fma(-t, (double)nseg, m) * inv;
    const double a = seg_mul(n, ls), b = seg_mul(t, dl);
    const double s = a + b, z = s - a;
    const double e = (a - (s - z)) + (b - z) + (fma(n, ls, -a) + fma(tl, dl, fma(t, dl, -b)));
    const double hi = seg_mul(s, c);
    return TwoDouble{hi, fma(e, c, fma(s, c, -hi))};
}

}  // namespace scdat
