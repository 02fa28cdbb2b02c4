// segment_cloud.h on the host: the points of the closed form are those a loop over all of them takes, and
// its sums, and those of a run of terms, are no further from the exact ones than terms rounded one by one
// and added exactly.
#include "segment_cloud.h"

#include <cstdio>
#include <random>

using namespace scdat;

constexpr double kEps = 1e-8;

static int check(const double* ls, const double* dl, int nseg)
{
    const SegPoints p = seg_points(ls, dl, nseg, kEps);
    int bad = 0;
    for (int k = 0; k < nseg; ++k)
        if (seg_inside(ls, dl, nseg, kEps, k) != (k >= p.first && k <= p.last)) bad = 1;
    return bad;
}

// |sum - exact| of the closed form and of terms rounded one by one, in units of the larger of the terms' sums
// (113-bit reference)
static void errors(const double* ls, const double* dl, SegPoints p, int nseg, double c, double& closed, double& looped,
                   double& run)
{
    closed = looped = run = 0.0;
    for (int i = 0; i < 4; ++i) {
        __float128 exact = 0, loop = 0, size = 0;
        TwoDouble added{0.0, 0.0};
        for (int k = p.first; k <= p.last; ++k) {
            const double term = c * fma(((double)k + 0.5) / (double)nseg, dl[i], ls[i]);
            const __float128 e = (__float128)c * ((__float128)ls[i] + ((__float128)k + 0.5Q) / nseg * (__float128)dl[i]);
            exact += e;
            loop += term;
            size += e < 0 ? -e : e;
            seg_add(added, term);
        }
        const TwoDouble s = seg_sum(ls[i], dl[i], p, nseg, c);
        const __float128 got = (__float128)s.hi + s.lo, r = (__float128)added.hi + added.lo;
        if (size == 0) continue;
        closed = std::fmax(closed, std::fabs((double)((got - exact) / size)));
        looped = std::fmax(looped, std::fabs((double)((loop - exact) / size)));
        run = std::fmax(run, std::fabs((double)((r - loop) / size)));
    }
}

int main()
{
    std::mt19937_64 rng(3);
    std::uniform_real_distribution<double> u(0.0, 1.0);
    const int segs[] = {1, 2, 7, 10, 64, 128};
    long cases = 0, bad = 0;
    double worst = 0.0, worst_loop = 0.0, worst_run = 0.0, sum = 0.0, sum_loop = 0.0;
    for (int it = 0; it < 400000; ++it) {
        const int nseg = segs[it % 6];
        // a point in or near the tet, on or near a face's or a vertex's tolerance band, and a step of any length
        double ls[4], dl[4];
        for (int i = 1; i < 4; ++i) {
            ls[i] = -0.5 + 1.5 * u(rng);
            dl[i] = (2.0 * u(rng) - 1.0) * std::pow(10.0, -20.0 * u(rng));
        }
        const int kind = it / 6 % 4, at = 1 + it / 24 % 3;
        if (kind == 1) ls[at] = -kEps + 1e-24 * std::floor(9.0 * u(rng) - 4.0);
        if (kind == 2) ls[at] = 1.0 + kEps + 2.220446049250313e-16 * std::floor(9.0 * u(rng) - 4.0);
        if (kind == 3) dl[at] = 0.0;
        if (kind == 2)  // near the vertex: the others in their bands
            for (int i = 1; i < 4; ++i)
                if (i != at) ls[i] = -kEps * u(rng), dl[i] = 0.0;
        ls[0] = 1.0 - ls[1] - ls[2] - ls[3];
        dl[0] = -dl[1] - dl[2] - dl[3];
        if (kind == 2) ls[0] = -kEps * u(rng), dl[0] = 0.0;
        bad += check(ls, dl, nseg);
        ++cases;
        const SegPoints p = seg_points(ls, dl, nseg, kEps);
        double c, l, r;
        errors(ls, dl, p, nseg, -1.6e-19 / nseg * 3e5, c, l, r);
        worst = std::fmax(worst, c);
        worst_run = std::fmax(worst_run, r);
        worst_loop = std::fmax(worst_loop, l);
        sum += c;
        sum_loop += l;
    }
    const double nan = std::nan("");
    const double ls[4] = {nan, 0.1, 0.1, 0.1}, dl[4] = {0.0, 0.1, 0.1, nan};
    bad += check(ls, dl, 10);
    std::printf("%ld cases, %ld wrong; largest error %.1e, rounded one by one %.1e, of a run %.1e; mean %.1e and %.1e\n", cases, bad,
                worst, worst_loop, worst_run, sum / cases, sum_loop / cases);
    // a run in two doubles loses a few 2^-106 of its terms' sizes, 2^-100 with room for 128 terms; the closed form
    // is to be no further off than rounding one by one, at worst and on average
    return bad != 0 || worst_run > 8e-31 || worst > worst_loop || sum > sum_loop;
}
