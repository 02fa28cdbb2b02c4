// segment_cloud.h on the host: the points of the closed form are those a loop over all of them takes.
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

int main()
{
    std::mt19937_64 rng(3);
    std::uniform_real_distribution<double> u(0.0, 1.0);
    const int segs[] = {1, 2, 7, 10, 64, 128};
    long cases = 0, bad = 0;
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
    }
    const double nan = std::nan("");
    const double ls[4] = {nan, 0.1, 0.1, 0.1}, dl[4] = {0.0, 0.1, 0.1, nan};
    bad += check(ls, dl, 10);
    std::printf("%ld cases, %ld wrong\n", cases, bad);
    return bad != 0;
}
