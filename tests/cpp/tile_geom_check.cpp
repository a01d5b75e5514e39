// Shared-memory layout of the tiled solves (tile_geom.h) and the packed offset
// test (offset_pack.h), checked on the host: every address the kernel forms
// for a geometry lies inside the system's storage, no two live values share
// one, 16-byte accesses are aligned, and the neighbour offsets' words are
// clear of every row stored before the last covariances are gathered.
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "../../hpgl_b200/csrc/offset_pack.h"
#include "../../hpgl_b200/csrc/tile_geom.h"

using namespace hpgl_b200;

static int bad = 0;
#define CHECK(c)                                                        \
    do {                                                                \
        if (!(c) && ++bad < 20) printf("line %d: %s\n", __LINE__, #c); \
    } while (0)

template <typename T>
static void geometry() {
    std::vector<int> owner(T::SIZE, -1);
    auto own = [&](int at, int who) {
        CHECK(at >= 0 && at < T::SIZE);
        if (at < 0 || at >= T::SIZE) return;
        CHECK(owner[at] == -1);
        owner[at] = who;
    };
    for (int i = 0; i < T::NC; ++i) {
        const int a = i / T::CL, s = i % T::CL, row = T::rbase(a) + s * T::rstride(a);
        CHECK(row % 2 == 0 && T::pivot(a) % 2 == 0);
        for (int c = 0; c < T::CL; ++c) {
            CHECK(T::chunk(c, a) % 2 == 0);
            // whole pairs from the (even) block on, as they are stored and read
            for (int b = a & ~1; b < T::NB; b += 2) {
                own(row + T::chunk(c, a) + b - (a & ~1), i);
                own(row + T::chunk(c, a) + b + 1 - (a & ~1), i);
            }
        }
        own(row + T::pivot(a), i);
        own(row + T::pivot(a) + 1, i);
        // the table form of the same addresses
        const int x = row - (a & ~1), y = T::spread(a), z = T::mask(a), w = T::shift(a);
        for (int k = i; k < T::NC; ++k)
            CHECK(x + (k % T::CL) * y + ((k % T::CL & z) >> w) + k / T::CL ==
                  row + T::chunk(k % T::CL, a) + k / T::CL - (a & ~1));
        // the chunks' 16-byte words of one position, on different banks
        for (int c = 0; c < T::CL; ++c)
            for (int d = 0; d < c; ++d) CHECK((T::chunk(c, a) - T::chunk(d, a)) / 2 % 8 != 0);
    }
    // neighbour offsets: inside, and in no row of a block before NBA; the last
    // gather runs before block NB - 2's rows are stored
    CHECK(T::NBAT % 2 == 0 && T::NBAT + T::NC <= T::SIZE && T::NBAT >= T::rbase(T::NBA));
    CHECK(T::NBA >= T::NB - 2);
    CHECK(T::STRIDE >= T::SIZE && T::STRIDE % 2 == 0 && T::WARP == T::STRIDE * (T::G - 1) + T::SIZE);
    CHECK(T::NC <= T::SIZE);
}

template <typename T>
static void square() {
    std::vector<int> owner(T::SIZE, -1);
    auto own = [&](int at, int who) {
        CHECK(at >= 0 && at < T::SIZE);
        if (at < 0 || at >= T::SIZE) return;
        CHECK(owner[at] == -1);
        owner[at] = who;
    };
    CHECK(T::SIZE % 2 == 0 && T::RS % 2 == 0 && T::CS % 2 == 0 && T::CR % 2 == 0 && T::COL % 2 == 0);
    CHECK(T::NN + 1 <= T::NR && T::NR <= T::NC && T::NN + 1 < T::NC && T::BCOL == T::NC - 1);
    CHECK(T::L * T::XN >= T::NN + 1);
    for (int i = 0; i < T::NR; ++i)
        for (int c = 0; c < T::CL; ++c) {
            CHECK(T::off(c) % 2 == 0);
            // whole pairs, as they are stored and read
            for (int b = 0; b < T::NBC; b += 2) {
                own(i * T::RS + T::off(c) + b, i);
                own(i * T::RS + T::off(c) + b + 1, i);
            }
            for (int k = c; k < T::NC; k += T::CL) CHECK(T::at(i, k) == i * T::RS + T::off(c) + k / T::CL);
            for (int d = 0; d < c; ++d) CHECK((T::off(c) - T::off(d)) / 2 % 8 != 0);
        }
    for (int q = 0; q < 2; ++q)
        for (int r = 0; r < T::RL; ++r)
            for (int a = 0; a < T::NBR; a += 2) {
                own(T::COL + q * T::RL * T::CR + r * T::CR + a, 1000);
                own(T::COL + q * T::RL * T::CR + r * T::CR + a + 1, 1000);
            }
    CHECK(T::COL + T::NN <= T::SIZE && T::NN + 1 <= T::COL);
}

static void packing() {
    std::mt19937 rng(1);
    auto pick = [&](int lo, int hi) { return lo + (int)(rng() % (unsigned)(hi - lo + 1)); };
    int packed = 0;
    for (int it = 0; it < 4000; ++it) {
        int reach[3], t[3];
        const int top = it % 3 == 0 ? 12 : it % 3 == 1 ? 200 : 1500;
        for (int a = 0; a < 3; ++a) {
            reach[a] = pick(0, top);
            t[a] = pick(0, reach[a] + (it & 1));
        }
        const OffsetPack p(reach, t);
        if (p.m == 0) continue;
        ++packed;
        for (int q = 0; q < 400; ++q) {
            int o[2][3], d[3];
            bool in = true;
            for (int a = 0; a < 3; ++a) {
                // the difference at, next to and far from the range's edges
                const int e = pick(0, 5);
                d[a] = e == 0 ? t[a] : e == 1 ? -t[a] : e == 2 ? t[a] + 1 : e == 3 ? -t[a] - 1 : pick(-reach[a], reach[a]);
                if (d[a] > reach[a]) d[a] = reach[a];
                if (d[a] < -reach[a]) d[a] = -reach[a];
                o[0][a] = pick(-1000, 1000);
                o[1][a] = o[0][a] - d[a];
                in &= d[a] <= t[a] && d[a] >= -t[a];
            }
            const int v = (int)((unsigned)p.pack(o[0][0], o[0][1], o[0][2]) - (unsigned)p.pack(o[1][0], o[1][1], o[1][2]));
            CHECK(p.in_range(v) == in);
        }
    }
    CHECK(packed > 1000);
    const int huge[3] = {4000, 1000, 1000};
    CHECK(OffsetPack(huge, huge).m == 0);
}

int main() {
    geometry<TileGeom<8, 4, 1, 2, 10>>();
    geometry<TileGeom<12, 4, 1, 4, 10>>();
    geometry<TileGeom<16, 4, 1, 2, 10>>();
    geometry<TileGeom<20, 4, 1, 2, 10>>();
    geometry<TileGeom<24, 4, 1, 2, 10>>();
    geometry<TileGeom<28, 4, 2, 4, 8>>();
    geometry<TileGeom<32, 4, 2, 4, 8>>();
    geometry<TileGeom<36, 4, 4, 4>>();
    geometry<TileGeom<40, 4, 4, 4>>();
    geometry<TileGeom<44, 4, 4, 6>>();
    geometry<TileGeom<48, 4, 4, 6>>();
    geometry<TileGeom<52, 4, 4, 4>>();
    geometry<TileGeom<56, 4, 4, 4>>();
    geometry<TileGeom<64, 8, 4, 4>>();
    square<CokGeom<8, 4, 1>>();
    square<CokGeom<12, 4, 1>>();
    square<CokGeom<16, 4, 2>>();
    square<CokGeom<20, 4, 2>>();
    square<CokGeom<24, 4, 2>>();
    square<CokGeom<28, 4, 4>>();
    square<CokGeom<32, 4, 4>>();
    square<CokGeom<36, 4, 4>>();
    square<CokGeom<40, 8, 4>>();
    square<CokGeom<44, 8, 4>>();
    square<CokGeom<48, 8, 4>>();
    packing();
    printf(bad ? "%d failures\n" : "ok\n", bad);
    return bad != 0;
}
