// Lane tiles and shared-memory layouts of small systems (tile_solve.cuh,
// cok_tile.cuh): plain constants, compiled for host and device.
#pragma once

#ifdef __CUDACC__
#define HPGL_TILE_HD __host__ __device__
#else
#define HPGL_TILE_HD
#endif

namespace hpgl_b200 {

// Layout of an NC-column system's rows (TileGeom), CL chunks a row: the doubles
// of a chunk of row block a, the chunks' spread (chunk c starts at c spread +
// its part of the gaps below), the gaps' total, and all rows before block a.
HPGL_TILE_HD constexpr int chunk_c(int nc, int cl, int a) { return (nc / cl - (a & ~1) + 1) / 2 * 2; }
HPGL_TILE_HD constexpr int gap_c(int nc, int cl, int a) {
    const int cs = chunk_c(nc, cl, a);
    return cl == 4 ? (cs % 16 == 0 ? 6 : 2) : cs % 8 == 0 ? 6 : 2;
}
HPGL_TILE_HD constexpr int rbase_c(int nc, int cl, int a) {
    int s = 0;
    for (int q = 0; q < a; ++q) s += cl * (cl * chunk_c(nc, cl, q) + gap_c(nc, cl, q));
    return s;
}

template <int NC_, int CL_, int RL_, int PB_, int SKEW_ = 8>
struct TileGeom {
    static constexpr int NC = NC_, CL = CL_, RL = RL_, PB = PB_, SKEW = SKEW_;
    static constexpr int L = CL * RL;          // lanes of a system
    static constexpr int G = 32 / L;           // systems of a warp
    static constexpr int NB = NC / CL;         // column blocks
    static constexpr int H = CL / RL;          // rows of a block per lane
    static constexpr int XN = (NC + L - 1) / L;  // rows (right-hand side) per lane
    static_assert(NC % CL == 0 && CL % RL == 0 && 32 % L == 0, "tile shape");

    // Storage of a system: rows 0..NC-1 of the upper triangle, row i (block
    // a = i / CL) as CL chunks, chunk c holding columns c, c + CL, ... from
    // block a (rounded down to even) on.  A lane's columns (or rows) of one
    // row are then contiguous, 16-byte aligned pairs.  Gaps of two doubles
    // between chunks keep the chunk starts on different 16-byte bank
    // groups, make consecutive rows' starts (the column reads of the back
    // substitution, one row per lane) walk through the banks, and hold
    // RN(1 / U(i,i)) and U(i,i).
    static_assert(CL == 4 || (CL == 8 && NB < 16), "the chunk offsets are conflict-free for 4 and 8 chunks");
    HPGL_TILE_HD static constexpr int cs(int a) { return chunk_c(NC, CL, a); }
    // chunk c starts at c spread(a) + (c & mask(a)) / (shift(a) ? 2 : 1)
    HPGL_TILE_HD static constexpr int spread(int a) { return CL == 4 && cs(a) % 16 == 0 ? cs(a) + 2 : cs(a); }
    HPGL_TILE_HD static constexpr int mask(int a) {
        return CL == 4 ? (cs(a) % 16 == 8 ? 2 : 0) : cs(a) % 8 == 0 ? 6 : cs(a) % 8 == 4 ? 4 : 0;
    }
    HPGL_TILE_HD static constexpr int shift(int a) { return CL == 8 && cs(a) % 8 == 4 ? 1 : 0; }
    HPGL_TILE_HD static constexpr int chunk(int c, int a) { return c * spread(a) + ((c & mask(a)) >> shift(a)); }
    HPGL_TILE_HD static constexpr int pivot(int a) {
        return CL == 4 && cs(a) % 16 == 0 ? cs(a)
               : mask(a) == 0             ? CL * cs(a)
               : mask(a) == 4             ? 4 * cs(a)
                                          : 2 * cs(a);
    }
    HPGL_TILE_HD static constexpr int rstride(int a) { return CL * cs(a) + gap_c(NC, CL, a); }
    HPGL_TILE_HD static constexpr int rbase(int a) { return rbase_c(NC, CL, a); }
    // The neighbour offsets (NC 8-byte words) lie in the last rows: those of
    // the last block, or of the last two.  The last block's covariances, the
    // last to be gathered, are gathered before the first row of the block
    // before it is stored.  The vectors of the outputs take the factor's place
    // afterwards.
    static constexpr int NBA = rbase_c(NC, CL, NB) - rbase_c(NC, CL, NB - 1) >= NC ? NB - 1 : NB - 2;
    static_assert(rbase_c(NC, CL, NB) - rbase_c(NC, CL, NBA) >= NC, "room for the neighbour offsets");
    static constexpr int NBAT = rbase_c(NC, CL, NBA);
    static constexpr int SIZE = rbase_c(NC, CL, NB);
    // Distance of two systems of a warp: 8-byte accesses go half a warp at a
    // time, so where several systems share such a pass they start SKEW
    // doubles apart in the banks.
    static constexpr int STRIDE = SIZE + (G > 2 ? ((SKEW - SIZE) % 16 + 16) % 16 : 0);
    static constexpr int WARP = STRIDE * (G - 1) + SIZE;
};

// The square of a cokriging system (cok_tile.cuh).
template <int NN_, int CL_, int RL_>
struct CokGeom {
    static constexpr int NN = NN_, CL = CL_, RL = RL_;  // NN: neighbours, even
    static constexpr int L = CL * RL, G = 32 / L, H = CL / RL;
    static constexpr int NBC = (NN + 2 + CL - 1) / CL;  // column blocks: NN + 1 unknowns, padding, B last
    static constexpr int NC = CL * NBC, BCOL = NC - 1;
    static constexpr int NBR = (NN + 1 + RL - 1) / RL;  // row blocks
    static constexpr int NR = RL * NBR;
    static constexpr int XN = (NN + 1 + L - 1) / L;     // unknowns per lane
    static_assert(NN % 2 == 0 && CL % RL == 0 && 32 % L == 0 && NC > NN + 1, "tile shape");
    // A row: CL chunks of CS doubles, chunk c the columns c, c + CL, ...; the
    // chunk starts on different 16-byte bank groups, rows two doubles apart
    static constexpr int even(int m) { return (m + 1) / 2 * 2; }
    static constexpr int CS = CL == 8 && even(NBC) % 4 == 0 ? even(NBC) + 2 : even(NBC);
    static constexpr int GAP = CL == 4 && CS % 16 == 8 ? 2 : 0;
    static constexpr int RS = CL * CS + 2;
    HPGL_TILE_HD static constexpr int off(int c) { return c * CS + (c & GAP); }
    HPGL_TILE_HD static constexpr int at(int i, int k) { return i * RS + off(k % CL) + k / CL; }
    // the pivot column, double buffered: chunk r the rows r, r + RL, ...; the
    // neighbour offsets lie there while the system is built
    static constexpr int CR = even(NBR) % 4 == 0 ? even(NBR) + 2 : even(NBR);
    static constexpr int COL = NR * RS;
    static constexpr int SIZE = COL + (2 * RL * CR > NN ? 2 * RL * CR : even(NN));
};

}  // namespace hpgl_b200
