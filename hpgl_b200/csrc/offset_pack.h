// A neighbour's offset from its node in one 32-bit word, and the test whether
// the difference of two offsets lies in the covariance table's range.
//
// The word is x + (y << sy) + (z << sz) in plain integer arithmetic, so the
// difference d of two words is the difference vector in the same form.  Each
// field is w bits wide with 2^(w-1) above the largest |difference| plus the
// range T of its axis; with k holding T + 2^(w-1) in every field, k + d and
// k - d hold v + T + 2^(w-1) and T - v + 2^(w-1), non-negative and below 2^w,
// so no field borrows from the next, and a field's top bit is set in both
// exactly when -T <= v <= T.  Three comparisons of three differences become
// one of the whole word.  m (the top bits) is 0 when the fields need more
// than 32 bits together: a field has two bits more than the largest power of
// two in reach + T.  The models that are cut at the search radii (T = the
// radii) pack up to several hundred cells on every axis; ordinary kriging and
// cokriging, whose T is about the reach, up to 256 cells on every axis, or more
// on one and fewer on the others, when the search spans them.
#pragma once

#ifdef __CUDACC__
#define HPGL_PACK_HD __host__ __device__ __forceinline__
#else
#define HPGL_PACK_HD inline
#endif

namespace hpgl_b200 {

struct OffsetPack {
    int sy = 0, sz = 0;
    unsigned k = 0, m = 0;
    OffsetPack() = default;
    // reach: the largest |difference| of two offsets per axis; t: the range
    OffsetPack(const int reach[3], const int t[3]) {
        int shift = 0;
        unsigned kk = 0, mm = 0;
        for (int a = 0; a < 3; ++a) {
            int w = 1;
            while (w < 32 && (1ll << (w - 1)) <= (long long)reach[a] + t[a]) ++w;
            if (shift + w > 32) return;
            if (a == 1) sy = shift;
            if (a == 2) sz = shift;
            kk += ((unsigned)t[a] + (1u << (w - 1))) << shift;
            mm |= 1u << (shift + w - 1);
            shift += w;
        }
        k = kk;
        m = mm;
    }
    HPGL_PACK_HD int pack(int x, int y, int z) const {
        return (int)((unsigned)x + ((unsigned)y << sy) + ((unsigned)z << sz));
    }
    HPGL_PACK_HD bool in_range(int d) const { return ((k + (unsigned)d) & (k - (unsigned)d) & m) == m; }
};

}  // namespace hpgl_b200
