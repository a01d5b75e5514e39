// Test driver: which jobs' neighbour offsets pack into one word
// (hpgl_b200/csrc/offset_pack.h), and the range test on the differences of
// packed offsets at and beyond the edges of every axis.
#include <cstdio>
#include <cstdlib>
#include <random>

#include "../../hpgl_b200/csrc/offset_pack.h"

using namespace hpgl_b200;

static int bad = 0;
#define CHECK(c)                                                   \
    do {                                                           \
        if (!(c) && bad++ < 20) printf("line %d: %s\n", __LINE__, #c); \
    } while (0)

static std::mt19937 g(7);
static int pick(int lo, int hi) { return lo + (int)(g() % (unsigned)(hi - lo + 1)); }

static void edges(const int reach[3], const int t[3], bool fits) {
    const OffsetPack p(reach, t);
    CHECK(p.fits == fits);
    if (!p.fits) return;
    for (int q = 0; q < 3000; ++q) {
        int o[2][3];
        bool in = true;
        for (int a = 0; a < 3; ++a) {
            const int e[] = {0, t[a], -t[a], t[a] + 1, -t[a] - 1, reach[a], -reach[a], pick(-reach[a], reach[a])};
            int d = e[pick(0, 7)];
            d = d > reach[a] ? reach[a] : d < -reach[a] ? -reach[a] : d;
            o[0][a] = pick(-(reach[a] + 1) / 2, (reach[a] + 1) / 2);
            o[1][a] = o[0][a] - d;
            in &= d <= t[a] && d >= -t[a];
        }
        const int v = (int)((unsigned)p.pack(o[0][0], o[0][1], o[0][2]) - (unsigned)p.pack(o[1][0], o[1][1], o[1][2]));
        CHECK(p.in_range(v) == in);
    }
}

int main() {
    // untruncated models: the table spans the differences, whatever the size
    const int spans[][3] = {{299, 299, 299}, {4096, 64, 64}, {1200, 1200, 1200}, {0, 0, 0}, {40000, 20000, 1}};
    for (auto &r : spans) edges(r, r, true);
    // cut at the radii: a quarter of the reach, half of it, all of it
    const int quarter[][3] = {{419, 419, 419}, {681, 681, 681}, {2730, 340, 340}};
    for (auto &r : quarter) {
        const int t[3] = {r[0] / 4, r[1] / 4, r[2] / 4};
        edges(r, t, true);
    }
    const int r511[3] = {511, 511, 511}, t255[3] = {255, 255, 255};
    edges(r511, t255, true);
    // two axes that no difference leaves, the third alone in the word
    const int wide[3] = {200000, 5000, 5000}, flat[3] = {50000, 5000, 6000};
    edges(wide, flat, true);
    // fields that need 33 bits
    const int r682[3] = {682, 682, 682}, t170[3] = {170, 170, 170};  // reach - t = 512
    edges(r682, t170, false);
    const int r513[3] = {513, 513, 513}, t256[3] = {256, 256, 256};  // 2 t = 512
    edges(r513, t256, false);
    for (int q = 0; q < 4000; ++q) {
        int r[3], t[3];
        for (int a = 0; a < 3; ++a) {
            r[a] = pick(0, q % 3 == 0 ? 20 : q % 3 == 1 ? 400 : 3000);
            t[a] = pick(0, r[a] + 1);
        }
        edges(r, t, OffsetPack(r, t).fits);
    }
    printf(bad ? "%d failures\n" : "ok\n", bad);
    return bad != 0;
}
