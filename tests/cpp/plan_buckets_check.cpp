// Test driver: the clusterizer buckets of a plan (hpgl_b200/csrc/plan.cpp,
// counted and filled strip by strip on all threads) against buckets filled
// here node by node in index order: starts, nodes, informed count.  Grids
// smaller than a box, boxes smaller than a cell row, odd sizes, dense and
// empty masks.  Returns the number of mismatching plans.
#include <random>
#include <vector>

#include "../../hpgl_b200/csrc/plan.h"

using namespace hpgl_b200;

extern "C" int pbc_run(unsigned seed, int cases, int threads) {
    std::mt19937 g(seed);
    int bad = 0;
    for (int t = 0; t < cases; ++t) {
        const int nx = 1 + g() % 90, ny = 1 + g() % 70, nz = 1 + g() % 30;
        const unsigned share[] = {0, 1, 20, 200, 1000};
        const unsigned per_mille = share[g() % 5];
        std::vector<uint8_t> m((size_t)nx * ny * nz);
        for (auto &x : m) x = g() % 1000 < per_mille;
        KrigingParams p{};
        p.cov_type = g() % 3;
        for (int a = 0; a < 3; ++a) {
            p.ranges[a] = 2 + g() % 20;
            p.radii[a] = 1 + g() % 25;
        }
        p.sill = 1;
        p.max_neighbours = 8;
        Plan P;
        build_plan(P, KIND_SK, nx, ny, nz, p, m.data(), threads, false);
        const long long nb = (long long)P.mx * P.my * P.mz;
        std::vector<std::vector<int>> box(nb);
        long long informed = 0;
        for (long long i = 0; i < P.size; ++i)
            if (m[i]) {
                const int x = (int)(i % nx), y = (int)(i / nx % ny), z = (int)(i / ((long long)nx * ny));
                box[((long long)(int)(z / P.cl_r[2]) * P.my + (int)(y / P.cl_r[1])) * P.mx + (int)(x / P.cl_r[0])].push_back((int)i);
                ++informed;
            }
        bool same = P.informed == informed && (long long)P.bucket_start.size() == nb + 1 && P.bucket_start[0] == 0;
        for (long long b = 0; same && b < nb; ++b) {
            if ((long long)box[b].size() > P.limit) box[b].clear();
            same = P.bucket_start[b + 1] - P.bucket_start[b] == (int)box[b].size();
            for (size_t k = 0; same && k < box[b].size(); ++k) same = P.bucket_nodes[P.bucket_start[b] + k] == box[b][k];
        }
        bad += !same;
    }
    return bad;
}
