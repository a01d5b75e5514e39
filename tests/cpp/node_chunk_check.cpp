// Test driver: the last chunks of grids up to the largest number of nodes
// (hpgl_b200/csrc/node_chunk.h): every node handed out once and no other, the
// counter running past the largest int as warps go on taking chunks.
#include <climits>
#include <cstdio>
#include <vector>

#include "../../hpgl_b200/csrc/node_chunk.h"

using namespace hpgl_b200;

int main() {
    int bad = 0;
    const long long sizes[] = {1, 31, 32, 33, 100000, INT_MAX - 70000LL, INT_MAX - 32LL, INT_MAX - 1LL, INT_MAX};
    for (long long size : sizes)
        for (int chunk : {1, 2, 7, 16, 32}) {
            const long long tail = size < 1000 ? size : 1000;
            std::vector<int> seen((size_t)tail, 0);
            unsigned counter = (unsigned)(size - tail);
            for (int warp = 0; warp < 12000; ++warp, counter += (unsigned)chunk) {
                const long long first = chunk_first((int)counter, size);
                if (first >= size) continue;
                for (int l = 0; l < 32; ++l) {
                    if (!chunk_has((int)first, l, chunk, size)) continue;
                    const long long node = (int)((unsigned)first + (unsigned)l);
                    if (node < size - tail || node >= size) ++bad;
                    else ++seen[(size_t)(node - (size - tail))];
                }
            }
            for (int s : seen) bad += s != 1;
        }
    printf(bad ? "%d failures\n" : "ok\n", bad);
    return bad != 0;
}
