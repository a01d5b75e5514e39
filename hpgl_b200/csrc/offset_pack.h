// A neighbour's offset from its node in one 32-bit word, and the test whether
// the difference of two offsets lies in the covariance table's range.
//
// The word holds a field of the tested axes in plain integer arithmetic, x +
// (y << shift) + ..., so the difference d of two words is the difference vector
// in the same form.  A field is w bits wide, H = 2^(w-1) above twice the axis's
// range T and above what the largest |difference| exceeds T by; k holds T + H in
// every field.  While the fields below are in range, a field of k + d is
// v + T + H and of k - d is T - v + H, each in [H, 2H) when -T <= v <= T, so
// that nothing carries into the next field; in the lowest field out of range
// one of the two is in [0, H) and its top bit clear.  So the top bits (m) are
// all set in both words exactly when every axis is in range: three comparisons
// of three differences become one of the whole word.
//
// Where the fields of all three axes need more than 32 bits, the axes whose
// range no difference can leave go without (m = 0, always in range, where no
// axis is left).  That takes in every job of the untruncated models (ordinary
// kriging, cokriging), whose table spans their differences; the models that are
// cut at the search radii pack up to about 680 cells on every axis with radii of
// a quarter of them, 512 with radii of half.  With fields above reach + T for
// all axes, as they were, 300x300x300 ordinary kriging with radii 75 did not
// pack and its 27 M systems of 32 neighbours took 373 ms one a warp where the
// tiles take 129, SK 420x420x420 with radii 105 (73 M) 933 where they take 308; a
// mixed request had taken 173 and 391 with the FP32 arithmetic that went.
#pragma once

#ifdef __CUDACC__
#define HPGL_PACK_HD __host__ __device__ __forceinline__
#else
#define HPGL_PACK_HD inline
#endif

namespace hpgl_b200 {

struct OffsetPack {
    unsigned mx = 0, my = 0, mz = 0;  // the axes' places in the word
    unsigned k = 0, m = 0;
    bool fits = false;
    OffsetPack() = default;
    // reach: the largest |difference| of two offsets per axis; t: the range
    OffsetPack(const int reach[3], const int t[3]) { fits = place(reach, t, true) || place(reach, t, false); }
    HPGL_PACK_HD int pack(int x, int y, int z) const {
        return (int)((unsigned)x * mx + (unsigned)y * my + (unsigned)z * mz);
    }
    HPGL_PACK_HD bool in_range(int d) const { return ((k + (unsigned)d) & (k - (unsigned)d) & m) == m; }

private:
    // all: also the axes that no difference leaves
    bool place(const int reach[3], const int t[3], bool all) {
        unsigned *at[3] = {&mx, &my, &mz};
        int shift = 0;
        k = m = mx = my = mz = 0;
        for (int a = 0; a < 3; ++a) {
            if (!all && t[a] >= reach[a]) continue;
            const long long most = 2ll * t[a] > (long long)reach[a] - t[a] ? 2ll * t[a] : (long long)reach[a] - t[a];
            int w = 1;
            while (w < 33 && (1ll << (w - 1)) <= most) ++w;
            if (shift + w > 32) {
                k = m = mx = my = mz = 0;
                return false;
            }
            *at[a] = 1u << shift;
            k += ((unsigned)t[a] + (1u << (w - 1))) << shift;
            m |= 1u << (shift + w - 1);
            shift += w;
        }
        return true;
    }
};

}  // namespace hpgl_b200
