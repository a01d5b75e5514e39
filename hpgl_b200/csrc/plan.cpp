// Host planning of a kriging job.  Compiled with -O2 -ffp-contract=off so
// that every covariance value is the one the reference computes (same
// expression order, glibc libm, no fused multiply-adds).  Paths cited are
// relative to the reference's src/geo_bsd/hpgl/.
#include "plan.h"

#include <algorithm>
#include <cstring>
#include <atomic>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <cmath>
#include <stdexcept>
#include <mutex>
#include <thread>

#include "introsort.h"
#include "task_pool.h"

namespace hpgl_b200 {



static std::atomic<int> g_threads{0};

int host_threads() {
    int n = g_threads.load();
    if (n > 0) return n;
    unsigned hc = std::thread::hardware_concurrency();
    return hc ? (int)hc : 1;
}

void set_host_threads(int n) { g_threads.store(n > 0 ? n : 0); }

// f(lo, hi) over [0, n) split across up to `threads` threads of the pool, at
// least `grain` items per thread.
template <typename F>
static void parallel_for(long long n, int threads, F f, long long grain = 4096) {
    pool_for(n, threads, f, grain);
}

// C(v) over the box |v_i| <= r_i into out[((z+rz)*(2ry+1) + y+ry)*(2rx+1) + x+rx],
// evaluated as f(x, y, z).  C(v) == C(-v) bit for bit (every transformed
// component only changes sign), so the half with z > 0 or (z == 0, y > 0) or
// (z == y == 0, x >= 0) is evaluated and mirrored.
template <typename V, typename F>
static void fill_symmetric(V &out, int rx, int ry, int rz, int threads, F f) {
    const int xd = 2 * rx + 1, yd = 2 * ry + 1;
    out.clear();
    out.resize((size_t)xd * yd * (2 * rz + 1));  // every entry is written below
    auto idx = [&](int x, int y, int z) { return ((size_t)(z + rz) * yd + (y + ry)) * xd + (x + rx); };
    // rows (z, y) of the evaluated half, z = 0..rz (y >= 0 at z = 0), a few
    // thousand covariances per thread at least
    const long long rows = (long long)(rz + 1) * yd;
    parallel_for(
        rows, threads,
        [&](long long lo, long long hi) {
            for (long long r = lo; r < hi; ++r) {
                const int z = (int)(r / yd), y = (int)(r % yd) - ry;
                if (z == 0 && y < 0) continue;
                for (int x = (z == 0 && y == 0 ? 0 : -rx); x <= rx; ++x) {
                    const double v = f(x, y, z);
                    out[idx(x, y, z)] = v;
                    out[idx(-x, -y, -z)] = v;
                }
            }
        },
        std::max<long long>(1, 4096 / xd));
}

// Sub-ranges above this many entries may go to another thread.
constexpr int SORT_SPAWN_MIN = 4096;

// sort_partition's result with fewer mispredicted branches (BlockQuicksort,
// Edelkamp and Weiss, ESA 2016): the positions of the left stoppers of a block
// of 64 at the low end and of the right stoppers of one at the high end are
// collected without branching, and the k-th left stopper is swapped with the
// k-th right stopper -- the pairs the scans of the Hoare partition meet one
// after the other.  Once fewer than two blocks are left between the ends,
// the scans themselves go on from the first unmatched stopper of each side
// (or from the end, where a block's stoppers are used up).
static int sort_partition_blocks(SortArr a, int lo, int hi, int pivot) {
    constexpr int BLOCK = 64;
    const double pk = a.key[pivot];
    uint8_t left[BLOCK], right[BLOCK];
    int nl = 0, nr = 0, sl = 0, sr = 0;
    while (hi - lo > 2 * BLOCK) {
        if (nl == 0) {
            sl = 0;
            for (int i = 0; i < BLOCK; ++i) {
                left[nl] = (uint8_t)i;
                nl += !(a.key[lo + i] > pk);
            }
        }
        if (nr == 0) {
            sr = 0;
            for (int i = 0; i < BLOCK; ++i) {
                right[nr] = (uint8_t)i;
                nr += !(pk > a.key[hi - 1 - i]);
            }
        }
        const int m = std::min(nl, nr);
        for (int k = 0; k < m; ++k) a.swap(lo + left[sl + k], hi - 1 - right[sr + k]);
        nl -= m;
        nr -= m;
        sl += m;
        sr += m;
        if (nl == 0) lo += BLOCK;
        if (nr == 0) hi -= BLOCK;
    }
    if (nl) lo += left[sl];
    if (nr) hi -= right[sr];
    return sort_partition(a, lo, hi, pivot);
}

// The reference's std::sort permutation (introsort.h) with the independent
// right-hand sub-ranges of large partitions sorted as pool tasks: each
// sub-range's processing touches only its own elements, so the result is
// the sequential algorithm's, element for element, whatever runs where.  The
// final insertion sort only moves elements within the runs of at most 16 that
// the partitioning leaves (no element of a later run comes before one of an
// earlier run), so each run is inserted as soon as it is reached, while it is
// in the cache, instead of by one pass over the whole array at the end; a
// heap-sorted range is already in order.
static void sort_subrange(SortArr a, int lo, int hi, int depth, TaskGroup &g) {
    while (hi - lo > 16) {
        if (depth == 0) {
            sort_heapsort(a, lo, hi);
            return;
        }
        --depth;
        const int mid = lo + (hi - lo) / 2;
        sort_median_to_first(a, lo, lo + 1, mid, hi - 1);
        const int cut = sort_partition_blocks(a, lo + 1, hi, lo);
        if (hi - cut > SORT_SPAWN_MIN)
            task_submit(g, [a, cut, hi, depth, &g] { sort_subrange(a, cut, hi, depth, g); });
        else
            sort_subrange(a, cut, hi, depth, g);
        hi = cut;
    }
    sort_insertion(a, lo, hi);
}

static void parallel_reference_sort(RawVector<double> &key, RawVector<int> &idx, int threads) {
    const int n = (int)key.size();
    if (n <= 1) return;
    SortArr a{key.data(), idx.data()};
    if (threads > 1) task_pool_reserve(threads - 1);
    TaskGroup g;
    std::exception_ptr own;
    try {
        sort_subrange(a, 0, n, 2 * sort_floor_log2(n), g);
    } catch (...) {
        own = std::current_exception();
    }
    task_wait(g);
    if (own) std::rethrow_exception(own);
}

// 3x3 product summed left to right, as TNT's matmult (tnt_cmat.h:472-498).
static void mat3(const double *a, const double *b, double *c) {
    for (int i = 0; i < 3; ++i)
        for (int k = 0; k < 3; ++k) {
            double s = 0;
            for (int j = 0; j < 3; ++j) s = s + a[3 * i + j] * b[3 * j + k];
            c[3 * i + k] = s;
        }
}

CovModel::CovModel(const KrigingParams &p) {
    type = p.cov_type;
    sill = p.sill;
    nugget = p.nugget;
    range0 = p.ranges[0];
    // create_transform (cov_model.h:16-61); grad_to_rad is (grad*pi)/180.
    const double pi = 3.14159265358979323846264338327950288419;
    const double a0 = (p.angles[0] * pi) / 180, a1 = (p.angles[1] * pi) / 180, a2 = (p.angles[2] * pi) / 180;
    const double s[9] = {1.0, 0, 0, 0, p.ranges[0] / p.ranges[1], 0, 0, 0, p.ranges[0] / p.ranges[2]};
    const double rz[9] = {cos(a0), sin(a0), 0, -sin(a0), cos(a0), 0, 0, 0, 1};
    const double ry[9] = {cos(a1), 0, -sin(a1), 0, 1, 0, sin(a1), 0, cos(a1)};
    const double rx[9] = {1, 0, 0, 0, cos(a2), sin(a2), 0, -sin(a2), cos(a2)};
    double xy[9], xyz[9];
    mat3(rx, ry, xy);
    mat3(xy, rz, xyz);
    mat3(s, xyz, t);
}

double CovModel::operator()(double vx, double vy, double vz) const {
    const double v[3] = {vx, vy, vz};
    double acc = 0.0;
    for (int i = 0; i < 3; ++i) {
        double d = 0.0;
        for (int j = 0; j < 3; ++j) d += v[j] * t[3 * i + j];
        acc += d * d;
    }
    const double h = sqrt(acc);
    if (h < 0.0001) return sill - nugget;
    switch (type) {
    case 2: return (sill - nugget) * exp(-3 * pow(h / range0, 2));
    case 1: return (sill - nugget) * exp(-3 * h / range0);
    default:
        if (h > range0) return 0;
        return (sill - nugget) * (1 - 1.5 * h / range0 + 0.5 * pow(h / range0, 3));
    }
}

// The clusterizer keeps candidates of C(d) > C(0)/100.  C falls with
// h = |T d|, so only h below the distance where the model falls to a hundredth
// can pass.  The limit has room for the roundings: 1e-3 of h for the model's,
// and for |T d| in single precision, whose terms may cancel, 1e-6 of the
// largest sum of their magnitudes (a sum of three products is off by at most 4
// roundings of 6e-8 each, the coefficients' included, per component).
static void cov_reach(const CovModel &cov, const int n[3], float t[9], float &limit) {
    double magnitude = 0;
    for (int i = 0; i < 9; ++i) {
        t[i] = (float)cov.t[i];
        magnitude += fabs(cov.t[i]) * n[i % 3];
    }
    limit = INFINITY;
    if (!(cov.sill - cov.nugget > 0) || !(cov.range0 > 0)) return;
    // spherical: 1 - 1.5 r + 0.5 r^3 = 0.01 at r = 0.9172; exponential: exp(-3 r);
    // Gaussian: exp(-3 r^2)
    const double r = cov.type == 2 ? sqrt(log(100.0) / 3) : cov.type == 1 ? log(100.0) / 3 : 0.918;
    const double h = cov.range0 * r * 1.001 + 0.001 + 1e-6 * magnitude;
    limit = (float)(h * h);
}

void validate_params(const KrigingParams &p, int kind) {
    if (p.cov_type < 0 || p.cov_type > 2) throw std::invalid_argument("covariance type must be 0, 1 or 2");
    for (int i = 0; i < 3; ++i) {
        // cov_model.h:24-25 raises on a zero range.
        if (p.ranges[i] == 0) throw std::invalid_argument("All covariance ranges should be non-zero");
        if (p.radii[i] <= 0) throw std::invalid_argument("search radiuses must be positive");
    }
    if (p.max_neighbours <= 0) throw std::invalid_argument("max_neighbours must be positive");
    if (p.max_neighbours > 64) throw std::domain_error("max_neighbours > 64 is not supported by this build");
    if (kind == KIND_IK && !(p.marginal_prob == p.marginal_prob))
        throw std::invalid_argument("marginal probability is NaN");
}

bool same_system(const KrigingParams &a, const KrigingParams &b) {
    if (a.cov_type != b.cov_type || a.sill != b.sill || a.nugget != b.nugget || a.max_neighbours != b.max_neighbours)
        return false;
    for (int i = 0; i < 3; ++i)
        if (a.ranges[i] != b.ranges[i] || a.angles[i] != b.angles[i] || a.radii[i] != b.radii[i]) return false;
    return true;
}

double informed_mean(const float *values, const uint8_t *mask, long long size) {
    int count = 0;
    double sum = 0;
    for (long long i = 0; i < size; ++i)
        if (mask[i]) {
            sum += values[i];
            count += 1;
        }
    return count == 0 ? 0 : sum / count;
}

// ---- clusterizer (clusterizer.cpp:52-184) ----
// Boxes of the radii (doubles in the reference: sugarbox_search_ellipsoid_t),
// mx = (int)(nx / rx + 2); a box overflows past limit = |template| / 250
// (sugarbox_indexed_neighbour_lookup.h:58) and then holds no nodes.  Fills
// P's clusterizer fields (P.size and P.clusterizer set).
static void build_buckets(Plan &P, int nx, int ny, int nz, const KrigingParams &p, const uint8_t *mask,
                          long long limit, int threads) {
    for (int i = 0; i < 3; ++i) P.cl_r[i] = (double)p.radii[i];
    P.mx = (int)(nx / P.cl_r[0] + 2);
    P.my = (int)(ny / P.cl_r[1] + 2);
    P.mz = (int)(nz / P.cl_r[2] + 2);
    P.limit = limit;
    const long long nb = (long long)P.mx * P.my * P.mz;
    std::vector<int> count(nb, 0);
    std::vector<uint8_t> exceeded(nb, 0);
    // A box takes the informed nodes in index order until it holds `limit`,
    // and the next one makes it overflow: it overflows exactly when it
    // receives more than `limit` nodes.  Boxes of one (y, z) strip hold the
    // nodes of one rectangle of grid rows, so the strips are counted and
    // filled independently, each row by row (which is index order), on all
    // threads.
    std::vector<int> bx(nx), ystrip(1, 0), zstrip(1, 0);  // box of x; first rows of the strips
    for (int x = 0; x < nx; ++x) bx[x] = (int)(x / P.cl_r[0]);
    std::vector<int> sy(1, 0), sz(1, 0);  // box of each strip
    for (int y = 1; y < ny; ++y) {
        const int b = (int)(y / P.cl_r[1]);
        if (b != sy.back()) {
            sy.push_back(b);
            ystrip.push_back(y);
        }
    }
    for (int z = 1; z < nz; ++z) {
        const int b = (int)(z / P.cl_r[2]);
        if (b != sz.back()) {
            sz.push_back(b);
            zstrip.push_back(z);
        }
    }
    ystrip.push_back(ny);
    zstrip.push_back(nz);
    const long long strips = (long long)sy.size() * (long long)sz.size();
    const long long grain = std::max<long long>(1, strips * 65536 / std::max<long long>(1, P.size));
    // f(x, index, first box of the strip) over a strip's informed nodes
    auto each_informed = [&](long long strip, auto f) {
        const int jy = (int)(strip % (long long)sy.size()), jz = (int)(strip / (long long)sy.size());
        const long long box = ((long long)sz[jz] * P.my + sy[jy]) * P.mx;
        for (int z = zstrip[jz]; z < zstrip[jz + 1]; ++z)
            for (int y = ystrip[jy]; y < ystrip[jy + 1]; ++y) {
                const long long row = ((long long)z * ny + y) * nx;
                const uint8_t *m = mask + row;
                int x = 0;
                for (; x + 8 <= nx; x += 8) {
                    uint64_t w;
                    memcpy(&w, m + x, 8);
                    if (!w) continue;
                    for (int k = 0; k < 8; ++k)
                        if (m[x + k]) f(x + k, (int)(row + x + k), box);
                }
                for (; x < nx; ++x)
                    if (m[x]) f(x, (int)(row + x), box);
            }
    };
    parallel_for(
        strips, threads,
        [&](long long lo, long long hi) {
            for (long long s = lo; s < hi; ++s) each_informed(s, [&](int x, int, long long box) { ++count[box + bx[x]]; });
        },
        grain);
    P.informed = 0;
    for (long long b = 0; b < nb; ++b) {
        P.informed += count[b];
        if (count[b] > P.limit) {
            exceeded[b] = 1;
            count[b] = 0;
        }
    }
    P.bucket_start.assign(nb + 1, 0);
    for (long long b = 0; b < nb; ++b) P.bucket_start[b + 1] = P.bucket_start[b] + count[b];
    P.bucket_nodes.assign(P.bucket_start[nb], 0);
    if (P.bucket_start[nb] > 0) {
        std::vector<int> fill(P.bucket_start.begin(), P.bucket_start.end() - 1);
        parallel_for(
            strips, threads,
            [&](long long lo, long long hi) {
                for (long long s = lo; s < hi; ++s)
                    each_informed(s, [&](int x, int index, long long box) {
                        if (!exceeded[box + bx[x]]) P.bucket_nodes[fill[box + bx[x]]++] = index;
                    });
            },
            grain);
    }
    P.bucket_clean.assign(nb, 0);
    P.any_clean = false;
    P.all_clean = true;
    P.max_candidates = 0;
    // Only boxes that hold grid nodes are ever asked (cx < nx/rx + 1 < mx).
    for (int cz = 0; cz < P.mz; ++cz)
        for (int cy = 0; cy < P.my; ++cy)
            for (int cx = 0; cx < P.mx; ++cx) {
                if ((double)cx * P.cl_r[0] >= nx || (double)cy * P.cl_r[1] >= ny || (double)cz * P.cl_r[2] >= nz)
                    continue;
                bool clean = true;
                int cand = 0;
                for (int k = cz - 1; k <= cz + 1; ++k)
                    for (int j = cy - 1; j <= cy + 1; ++j)
                        for (int i = cx - 1; i <= cx + 1; ++i) {
                            if (i < 0 || j < 0 || k < 0 || i > P.mx || j > P.my || k > P.mz) continue;
                            long long b = ((long long)k * P.my + j) * P.mx + i;
                            if (b >= nb) continue;  // the inclusive box edge is never reached by real nodes
                            if (exceeded[b]) clean = false;
                            cand += count[b];
                        }
                long long b = ((long long)cz * P.my + cy) * P.mx + cx;
                if (!P.clusterizer) clean = false;
                P.bucket_clean[b] = clean ? 1 : 0;
                if (clean) {
                    P.any_clean = true;
                    P.max_candidates = std::max(P.max_candidates, cand);
                } else {
                    P.all_clean = false;
                }
            }

}

void build_plan(Plan &P, int kind, int nx, int ny, int nz, const KrigingParams &p, const uint8_t *mask,
                int threads, bool sequential) {
    static const bool timing = getenv("HPGL_B200_PLAN_TIMING") != nullptr;
    auto t_last = std::chrono::steady_clock::now();
    auto lap = [&](const char *what) {
        if (!timing) return;
        auto now = std::chrono::steady_clock::now();
        fprintf(stderr, "plan %-10s %8.2f ms\n", what, std::chrono::duration<double, std::milli>(now - t_last).count());
        t_last = now;
    };
    validate_params(p, kind);
    CovModel cov(p);
    P.kind = kind;
    P.nx = nx;
    P.ny = ny;
    P.nz = nz;
    P.size = (long long)nx * ny * nz;
    P.nmax = p.max_neighbours;
    // Ordinary kriging and cokriging use the model itself; cokriging searches
    // with neighbour_lookup_t alone (simple_cokriging_markI.cpp:201, no
    // clusterizer).
    P.truncated = (kind != KIND_OK && !kind_is_cokriging(kind)) || sequential;
    P.clusterizer = !kind_is_cokriging(kind) && !sequential;
    for (int i = 0; i < 3; ++i) P.radii[i] = p.radii[i];
    const int rx = p.radii[0], ry = p.radii[1], rz = p.radii[2];

    // ---- search template: calc_cov_field (covariance_field.h:62-106) ----
    // C(0 - v) over the +-radius box in z-y-x order, offsets above C(0)/100
    // kept as the vector -v, sorted descending by std::sort (the same
    // unstable algorithm on the same input order as the reference, hence the
    // same order of equal keys).  Every covariance object the reference can
    // pass here (the model, the precalculated table, covariance_field_t)
    // yields these same values inside the box.
    const int xd = 2 * rx + 1, yd = 2 * ry + 1;
    RawVector<double> data;
    fill_symmetric(data, rx, ry, rz, threads, [&](int x, int y, int z) { return cov(0.0 - x, 0.0 - y, 0.0 - z); });
    lap("box");
    const double c0 = cov(0.0, 0.0, 0.0);
    const double threshold = c0 / 100;
    // Offsets -v in z-y-x order of v, keyed by C(v) (= C(-v)): counted per
    // z-slab in parallel (with the template's extent, that of the offsets above
    // the threshold), then written at the slabs' places.
    RawVector<double> keys;
    RawVector<int> order;
    P.ext[0] = P.ext[1] = P.ext[2] = 0;
    {
        const int zd = 2 * rz + 1;
        const long long plane = (long long)xd * yd, grain = std::max<long long>(1, 4096 / plane);
        std::vector<size_t> start((size_t)zd + 1, 0);
        std::vector<int> ez((size_t)zd * 3, 0);
        parallel_for(
            zd, threads,
            [&](long long lo, long long hi) {
                for (long long zi = lo; zi < hi; ++zi) {
                    int ex = 0, ey = 0;
                    size_t count = 0;
                    for (int y = -ry; y <= ry; ++y) {
                        const double *row = data.data() + zi * plane + (size_t)(y + ry) * xd;
                        size_t in_row = 0;
                        int first = xd, last = 0;
                        for (int x = 0; x < xd; ++x)
                            if (row[x] > threshold) {
                                ++in_row;
                                if (first == xd) first = x;
                                last = x;
                            }
                        if (in_row) {
                            ex = std::max(ex, std::max(std::abs(first - rx), std::abs(last - rx)));
                            ey = std::max(ey, std::abs(y));
                            count += in_row;
                        }
                    }
                    start[zi + 1] = count;
                    ez[3 * zi] = ex;
                    ez[3 * zi + 1] = ey;
                    ez[3 * zi + 2] = count ? std::abs((int)zi - rz) : 0;
                }
            },
            grain);
        for (int zi = 0; zi < zd; ++zi) {
            start[zi + 1] += start[zi];
            for (int a = 0; a < 3; ++a) P.ext[a] = std::max(P.ext[a], ez[3 * zi + a]);
        }
        keys.resize(start[zd]);
        order.resize(start[zd]);
        parallel_for(
            zd, threads,
            [&](long long lo, long long hi) {
                for (long long zi = lo; zi < hi; ++zi) {
                    const int z = (int)zi - rz;
                    size_t at = start[zi];
                    for (int y = -ry; y <= ry && at < start[zi + 1]; ++y) {
                        const double *row = data.data() + zi * plane + (size_t)(y + ry) * xd;
                        for (int x = -rx; x <= rx; ++x)
                            if (row[x + rx] > threshold) {
                                keys[at] = row[x + rx];
                                order[at++] = (int)((((size_t)(-z + rz) * yd) + (-y + ry)) * xd + (-x + rx));
                            }
                    }
                }
            },
            grain);
    }
    lap("keys");
    // Every collected key is above the threshold, so the template keeps all
    // of them and the clusterizer's limit (|template| / 250) is known before
    // the sort: the buckets are built as a pool task meanwhile.
    TaskGroup bucket_task;
    task_pool_reserve(1);
    task_submit(bucket_task, [&] { build_buckets(P, nx, ny, nz, p, mask, (long long)(keys.size() / 250), threads); });
    try {
        parallel_reference_sort(keys, order, threads);
    } catch (...) {
        try {
            task_wait(bucket_task);
        } catch (...) {
        }
        throw;
    }
    lap("sort");
    size_t kept = keys.size();
    for (size_t i = 0; i < keys.size(); ++i)
        if (keys[i] < threshold) {
            kept = i;
            break;
        }
    P.tmpl.resize(kept);
    parallel_for((long long)kept, threads, [&](long long lo, long long hi) {
        for (long long i = lo; i < hi; ++i) {
            const int o = order[i];
            TemplateEntry &e = P.tmpl[i];
            e.dx = o % xd - rx;
            e.dy = o / xd % yd - ry;
            e.dz = o / xd / yd - rz;
            e.delta = e.dx + nx * (e.dy + ny * e.dz);
        }
    });
    if (kept < keys.size()) {
        // entries cut after the sort (not reachable with the > threshold
        // filter, kept for the reference's second cut-off) do not widen ext
        P.ext[0] = P.ext[1] = P.ext[2] = 0;
        for (const TemplateEntry &e : P.tmpl) {
            P.ext[0] = std::max(P.ext[0], std::abs(e.dx));
            P.ext[1] = std::max(P.ext[1], std::abs(e.dy));
            P.ext[2] = std::max(P.ext[2], std::abs(e.dz));
        }
    }

    lap("template");
    task_wait(bucket_task);
    if ((long long)(P.tmpl.size() / 250) != P.limit)
        build_buckets(P, nx, ny, nz, p, mask, (long long)(P.tmpl.size() / 250), threads);
    lap("buckets");
    // ---- covariance table ----
    // Truncated kinds read C(v) only for |v| <= radii.  Ordinary kriging uses
    // the untruncated model; the template path needs |v| <= 2*ext (pairs of
    // template offsets), the clusterizer path |v| <= 4r-2 (pairs of
    // candidates from the 3x3x3 boxes).  No offset exceeds the grid.
    const int n3[3] = {nx, ny, nz};
    for (int a = 0; a < 3; ++a) {
        int need;
        if (P.truncated) {
            need = p.radii[a];
        } else {
            need = 2 * P.ext[a];
            if (P.any_clean) need = std::max(need, 4 * p.radii[a] - 2);
        }
        P.B[a] = std::max(0, std::min(need, n3[a] - 1));
        P.trunc[a] = P.truncated ? p.radii[a] : P.B[a];
    }
    if (P.B[0] == rx && P.B[1] == ry && P.B[2] == rz) {
        // the template's box already holds C(-v) at v, which is C(v) bit for
        // bit (the transform of -v is the negated transform of v, and only
        // its squares enter the distance)
        P.table.swap(data);
    } else {
        fill_symmetric(P.table, P.B[0], P.B[1], P.B[2], threads,
                       [&](int x, int y, int z) { return cov((double)x, (double)y, (double)z); });
    }
    P.c0 = c0;
    cov_reach(cov, n3, P.reach_t, P.reach_limit);
    lap("table");

    // ---- informed-bit rows for the device template search ----
    P.px = 32 * ((P.ext[0] + 31) / 32);
    P.nseg = (nx + 31) / 32;
    P.wpr = P.nseg + 2 * (P.px / 32) + 2;

}


void fill_cov_table(std::vector<double> &table, const int B[3], const KrigingParams &p, int threads) {
    CovModel cov(p);
    fill_symmetric(table, B[0], B[1], B[2], threads,
                   [&](int x, int y, int z) { return cov((double)x, (double)y, (double)z); });
}

}  // namespace hpgl_b200
