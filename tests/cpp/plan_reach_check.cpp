// Test driver: the offsets a plan lets pass to the covariance filter of the
// clusterizer search (cov_reach in hpgl_b200/csrc/plan.cpp) against the model.
// Every offset of the boxes around a node whose covariance exceeds C(0)/100
// must lie within reach_limit, the distance computed in single precision with
// and without fused multiply-adds; and the limit must not lie so far out that
// it drops nothing it could: offsets beyond it by 2 % and a cell are dropped.
// Returns the number of failing models; *kept and *dropped count offsets.
#include <cmath>
#include <random>

#include "../../hpgl_b200/csrc/plan.h"

using namespace hpgl_b200;

static float reach2(const Plan &P, float x, float y, float z, bool fused) {
    float q = 0.f;
    for (int i = 0; i < 3; ++i) {
        const float *t = P.reach_t + 3 * i;
        volatile float a = t[0] * x, b = t[1] * y, c = t[2] * z;
        if (fused) {
            const float u = fmaf(t[2], z, fmaf(t[1], y, a));
            q = fmaf(u, u, q);
        } else {
            volatile float ab = a + b;
            volatile float u = ab + c;
            volatile float uu = u * u;
            q = q + uu;
        }
    }
    return q;
}

extern "C" int prc_run(unsigned seed, int cases, long long *kept, long long *dropped) {
    std::mt19937 g(seed);
    auto pick = [&](double lo, double hi) { return lo * std::pow(hi / lo, g() / 4294967296.0); };
    int bad = 0;
    *kept = *dropped = 0;
    for (int t = 0; t < cases; ++t) {
        KrigingParams p{};
        p.cov_type = t % 3;
        const bool extreme = t % 4 == 3;
        int n[3];
        for (int a = 0; a < 3; ++a) {
            p.ranges[a] = extreme ? pick(0.001, 20000) : pick(1.5, 30);
            p.radii[a] = 1 + g() % 12;
            p.angles[a] = t % 5 ? g() % 360 : 0;
            n[a] = 2 * p.radii[a] + g() % 8;
        }
        p.sill = pick(1e-3, 1e3);
        p.nugget = t % 2 ? 0.3 * p.sill : 0;
        p.max_neighbours = 8;
        std::vector<uint8_t> m((size_t)n[0] * n[1] * n[2], 0);
        Plan P;
        build_plan(P, KIND_OK, n[0], n[1], n[2], p, m.data(), 1, false);
        const CovModel cov(p);
        const double c0 = cov(0, 0, 0);
        bool ok = true;
        for (int z = 1 - n[2]; z < n[2]; ++z)
            for (int y = 1 - n[1]; y < n[1]; ++y)
                for (int x = 1 - n[0]; x < n[0]; ++x) {
                    const bool pass = cov(x, y, z) > c0 / 100;
                    bool in = true;
                    for (int f = 0; f < 2; ++f)
                        in = in && !(reach2(P, (float)x, (float)y, (float)z, f) > P.reach_limit);
                    if (pass && !in) ok = false;
                    if (pass) ++*kept;
                    if (!in) ++*dropped;
                    if (!extreme && in && !pass) {
                        // not more than 2 % and a cell outside the model's own cut
                        const double s = 1.0 / 1.02;
                        const double far = cov(x * s, y * s, z * s);
                        if (!(far > c0 / 100) && std::sqrt((double)reach2(P, x, y, z, false)) > 1 &&
                            std::sqrt((double)P.reach_limit) > 1)
                            ok = false;
                    }
                }
        bad += !ok;
    }
    return bad;
}
