// FP64 factorisation and solution of small systems in the reference's exact
// operation order (my_kriging_weights.h:26-255 over LAPACK DPOTF2 / DPOTRS),
// several systems per warp, each spread over a two-dimensional cyclic tile of
// lanes.
//
// Measured on SK 256x256x64 (4.15 M systems of 32 neighbours): 17.5 ms where
// one column per lane and one system a warp took 53.2 ms.  ncu on the
// 128x128x32 cube: 2 251 instructions a system (8 387), FP64 pipe 31.8 %, the
// shared-memory / L1 data pipe 61.5 %, 8 warps an SM (their registers hold the
// accumulators): the pivot chain's latency and the L1 pipe bound it now.
//
// What bounds a small Cholesky factorisation is not its arithmetic: every
// step has a chain (pivot, square root, reciprocal, the row's scaling, its
// exchange between the lanes) that costs the same few dozen instructions
// whether one system or several go through it, and with one column per lane
// each lane reads the whole pivot row for one column's worth of products.
// Here a system takes L = CL x RL lanes; lane (r, c) accumulates the products
// of rows k = r mod RL and columns k = c mod CL, so a step reads
// (NB + H NB) values for H NB (NB+1)/2 products instead of one value per
// product, the open part shrinks evenly over the lanes, and 32 / L systems
// share every instruction of the chain.
//
// Bits: the sums t(i,k) = sum_{j<i} U(j,i) U(j,k) run over j in ascending
// order from +0 with separately rounded products, exactly as DDOT and DGEMV
// form them; they are merely all kept open (right-looking) instead of being
// formed one row at a time.  Entries of the padding beyond n are the
// identity's, so they add exact zeros nowhere near the live rows.
#pragma once
#include "device_common.cuh"
#include "search_common.cuh"
#include "tile_geom.h"

namespace hpgl_b200 {

// Per-block table of row i: U(i, k) = U[x + chunk(k % CL) + k / CL], with the
// chunk's offset (k % CL) y + ((k % CL & z) >> w).
template <typename T>
struct alignas(16) TileTables {
    short4 row[T::NC];
    __device__ void fill(int thread, int threads) {
        for (int i = thread; i < T::NC; i += threads) {
            const int a = i / T::CL;
            row[i] = make_short4((short)(T::rbase(a) + (i % T::CL) * T::rstride(a) - (a & ~1)),
                                 (short)T::spread(a), (short)T::mask(a), (short)T::shift(a));
        }
    }
    // chunk c of row q
    static __device__ __forceinline__ int chunk(const short4 &q, int c) {
        return c * q.y + (T::CL == 4 ? c & q.z : (c & q.z) >> q.w);
    }
};

// RN(sqrt(a)) and RN(1 / RN(sqrt(a))) together, without a branch:
// Goldschmidt's coupled iteration for sqrt(a) and 1 / (2 sqrt(a)) from the
// hardware's approximate reciprocal square root, then corrections by exact
// residuals (Markstein, IBM J. Res. Dev. 34(1), 1990): with g within an ulp of
// the root, a - g g is exact in one fused operation and g + (a - g g) h rounds
// correctly; with y within an ulp of 1 / s, y + (1 - s y) y rounds correctly
// unless s's significand is all ones and y lies below 1 / s, which the
// rounding up of the step before excludes.  Equal to __dsqrt_rn and __drcp_rn
// bit for bit for 2^-767 <= a < 2^769 (tests/test_tile_solve.py); a <= 0 or
// NaN, a singular system, gives what nobody reads.
__device__ __forceinline__ void sqrt_rcp(double a, double &root, double &rcp) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
    double g = __dmul_rn(a, y), h = __dmul_rn(0.5, y);
    double e = __fma_rn(-h, g, 0.5);
    g = __fma_rn(g, e, g);
    h = __fma_rn(h, e, h);
    e = __fma_rn(-h, g, 0.5);
    g = __fma_rn(g, e, g);
    h = __fma_rn(h, e, h);
    root = __fma_rn(__fma_rn(-g, g, a), h, g);
    y = __dadd_rn(h, h);
    y = __fma_ru(__fma_rn(-root, y, 1.0), y, y);
    rcp = __fma_rn(__fma_rn(-root, y, 1.0), y, y);
}

// Entries A(i, k) = C(x_i - x_k) (my_kriging_weights.h:49-58; the tables are
// exactly symmetric, C(v) = C(-v) bit for bit, so either orientation gives the
// reference's value) of the lane's rows
// of block p at its columns from block p on; the identity beyond n.
template <typename T>
__device__ __forceinline__ void tile_gather(const DevJob &J, const DevPlan &P, const int2 *nb, int n, int r,
                                            int c, int p, double (&a)[T::H][T::NB + 1]) {
    bool out = false;
#pragma unroll
    for (int h = 0; h < T::H; ++h) {
        const int i = T::CL * p + r + T::RL * h;
        const int2 o = nb[i];
#pragma unroll
        for (int b = 0; b < T::NB; ++b) {
            if (b < p) continue;
            const int k = T::CL * b + c;
            const int2 q = nb[k];
            const bool live = i < n && k < n, in = P.pk.in_range((int)((unsigned)o.x - (unsigned)q.x));
            a[h][b] = i == k ? 1.0 : 0.0;
            if (live && in) a[h][b] = __ldg(P.table + abs(o.y - q.y));
            out |= live && !in;
        }
    }
    if (out && !P.truncated) atomicOr(J.err, DERR_TABLE_RANGE);
}

// Factorises the warp's systems (DPOTF2 'U') and solves A x = b (and, for
// ordinary kriging, A x = 1) in DPOTRS's order; x[t] is row l + L t.  nw: the
// largest neighbour count of the warp's systems.  Returns whether the group's
// system is singular (its x is then meaningless).  A positive pivot is at
// least about 2^-54 C(0), so with C(0) in [PIVOT_C0_MIN, PIVOT_C0_MAX) it is in
// sqrt_rcp's range (tile_takes).
//
// Within a block of CL rows the products of a finished row with the rows of
// later blocks wait until the next row's pivot chain runs, so that the two
// share the issue slots; only the block's own rows are brought up to date at
// once.
template <typename T, bool ORD>
__device__ __forceinline__ bool tile_solve(const DevJob &J, const DevPlan &P, double *U, const TileTables<T> &B,
                                          int n, int nw, int l, double (&xa)[T::XN], double (&xb)[T::XN]) {
    constexpr int NB = T::NB, CL = T::CL, RL = T::RL, L = T::L, H = T::H, XN = T::XN;
    const int r = l / CL, c = l % CL;
    const int2 *nb = reinterpret_cast<const int2 *>(U + T::NBAT);
    double acc[H][NB + 1][NB];
    double u[NB + 1], w[H][NB + 1];  // the last finished row at the lane's columns and rows
#pragma unroll
    for (int h = 0; h < H; ++h)
#pragma unroll
        for (int p = 0; p < NB; ++p) {
            w[h][p] = 0.0;
#pragma unroll
            for (int b = p; b < NB; ++b) acc[h][p][b] = 0.0;
        }
#pragma unroll
    for (int b = 0; b <= NB; ++b) u[b] = 0.0;
    bool fail = false;
    // the covariances of a block's rows are gathered one block ahead
    double a[2][H][NB + 1];
    tile_gather<T>(J, P, nb, n, r, c, 0, a[0]);
#pragma unroll
    for (int p0 = 0; p0 < NB; ++p0) {
        // no open system, or only ones that have failed
        if (__all_sync(FULL_MASK, fail || n <= CL * p0)) break;
        const int PE = (p0 / T::PB + 1) * T::PB < NB ? (p0 / T::PB + 1) * T::PB : NB;  // the panel's end
        if (p0 > 0 && p0 % T::PB == 0) {
            // a panel's first block: the products of all finished rows
#pragma unroll 2
            for (int j = 0; j < CL * p0; ++j) {
                const short4 q = B.row[j];
                const double *colp = U + q.x + B.chunk(q, c);
                double cu[NB + 1];
#pragma unroll
                for (int b = p0; b < NB; b += 2) {
                    const double2 g = *reinterpret_cast<const double2 *>(colp + b);
                    cu[b] = g.x;
                    cu[b + 1] = g.y;
                }
#pragma unroll
                for (int h = 0; h < H; ++h) {
                    const double *rowp = U + q.x + B.chunk(q, r + RL * h);
#pragma unroll
                    for (int p = p0; p < PE; p += 2) {
                        const double2 g = *reinterpret_cast<const double2 *>(rowp + p);
#pragma unroll
                        for (int b = p; b < NB; ++b)
                            acc[h][p][b] = __dadd_rn(acc[h][p][b], __dmul_rn(g.x, cu[b]));
                        if (p + 1 < PE) {
#pragma unroll
                            for (int b = p + 1; b < NB; ++b)
                                acc[h][p + 1][b] = __dadd_rn(acc[h][p + 1][b], __dmul_rn(g.y, cu[b]));
                        }
                    }
                }
            }
#pragma unroll
            for (int h = 0; h < H; ++h)
#pragma unroll
                for (int p = p0; p < PE; ++p) w[h][p] = 0.0;
        }
        if (p0 + 1 < NB) tile_gather<T>(J, P, nb, n, r, c, p0 + 1, a[(p0 + 1) & 1]);
        if (p0 == T::NBA) __syncwarp();  // the rows that hold nb are stored from here on
#pragma unroll
        for (int h0 = 0; h0 < H; ++h0) {
#pragma unroll 1
            for (int rr = 0; rr < RL; ++rr) {
                const int s = h0 * RL + rr;  // row i = CL p0 + s
                double *row = U + T::rbase(p0) + s * T::rstride(p0);
                // the row's entries at the lane's columns (the row's owners:
                // the lanes of r == rr)
                double v[NB + 1];
#pragma unroll
                for (int b = p0; b < NB; ++b) v[b] = __dsub_rn(a[p0 & 1][h0][b], acc[h0][p0][b]);
                v[NB] = 0.0;
                const double ajj = __shfl_sync(FULL_MASK, v[p0], rr * CL + s, L);
                // the products that waited
#pragma unroll
                for (int h = 0; h < H; ++h)
#pragma unroll
                    for (int p = p0 + 1; p < PE; ++p)
#pragma unroll
                        for (int b = p; b < NB; ++b)
                            acc[h][p][b] = __dadd_rn(acc[h][p][b], __dmul_rn(w[h][p], u[b]));
                fail |= !(ajj > 0.0);
                double ujj, rinv;
                sqrt_rcp(ajj, ujj, rinv);
                if (r == rr) {
                    double *to = row + T::chunk(c, p0);
                    double q0 = __dmul_rn(rinv, v[p0]);
                    if (c == s) q0 = ujj;
                    if (p0 & 1) to[1] = q0;
#pragma unroll
                    for (int b = (p0 + 1) & ~1; b < NB; b += 2) {
                        double2 q = make_double2(__dmul_rn(rinv, v[b]), __dmul_rn(rinv, v[b + 1]));
                        if (b == p0) q.x = q0;
                        *reinterpret_cast<double2 *>(to + b - (p0 & ~1)) = q;
                    }
                }
                // forward substitution U^T y = b, dot form: row i is final
                const int xl = (CL * p0) % L + s;
                const double ya = div_by_rcp(__shfl_sync(FULL_MASK, xa[CL * p0 / L], xl, L), ujj, rinv);
                double yb = 0.0;
                if (ORD) yb = div_by_rcp(__shfl_sync(FULL_MASK, xb[CL * p0 / L], xl, L), ujj, rinv);
                if (l == xl) {
                    xa[CL * p0 / L] = ya;
                    if (ORD) xb[CL * p0 / L] = yb;
                    *reinterpret_cast<double2 *>(row + T::pivot(p0)) = make_double2(rinv, ujj);
                }
                __syncwarp();
                const double2 *colp = reinterpret_cast<const double2 *>(row + T::chunk(c, p0));
#pragma unroll
                for (int b = p0 & ~1; b < NB; b += 2) {
                    const double2 q = colp[(b - (p0 & ~1)) / 2];
                    u[b] = q.x;
                    u[b + 1] = q.y;
                }
#pragma unroll
                for (int h = 0; h < H; ++h) {
                    const double2 *rowp = reinterpret_cast<const double2 *>(row + T::chunk(r + RL * h, p0));
#pragma unroll
                    for (int p = p0 & ~1; p < PE; p += 2) {
                        const double2 q = rowp[(p - (p0 & ~1)) / 2];
                        w[h][p] = q.x;
                        w[h][p + 1] = q.y;
                    }
#pragma unroll
                    for (int b = p0; b < NB; ++b)
                        acc[h][p0][b] = __dadd_rn(acc[h][p0][b], __dmul_rn(w[h][p0], u[b]));
                }
#pragma unroll
                for (int t = 0; t < XN; ++t) {
                    if (L * (t + 1) <= CL * p0) continue;
                    if (l + L * t > CL * p0 + s && l + L * t < T::NC) {
                        const double q = row[T::chunk(c, p0) + r + RL * t - (p0 & ~1)];
                        xa[t] = __dsub_rn(xa[t], __dmul_rn(q, ya));
                        if (ORD) xb[t] = __dsub_rn(xb[t], __dmul_rn(q, yb));
                    }
                }
            }
        }
        // the next block's rows take the last row's products now
        if (p0 + 1 < PE) {
#pragma unroll
            for (int h = 0; h < H; ++h)
#pragma unroll
                for (int b = p0 + 1; b < NB; ++b)
                    acc[h][p0 + 1][b] = __dadd_rn(acc[h][p0 + 1][b], __dmul_rn(w[h][p0 + 1], u[b]));
        }
    }
    // U x = y, column form
    short4 at[XN];
#pragma unroll
    for (int t = 0; t < XN; ++t) at[t] = l + L * t < T::NC ? B.row[l + L * t] : make_short4(0, 0, 0, 0);
#pragma unroll
    for (int p0 = NB - 1; p0 >= 0; --p0) {
        if (CL * p0 >= nw) continue;
#pragma unroll 1
        for (int s = CL - 1; s >= 0; --s) {
            const int k = CL * p0 + s;
            const int xl = (CL * p0) % L + s;
            const double2 piv = *reinterpret_cast<const double2 *>(U + T::rbase(p0) + s * T::rstride(p0) + T::pivot(p0));
            double va = __shfl_sync(FULL_MASK, xa[CL * p0 / L], xl, L);
            const bool nza = va != 0.0;
            if (nza) va = div_by_rcp(va, piv.y, piv.x);
            double vb = 0.0;
            bool nzb = false;
            if (ORD) {
                vb = __shfl_sync(FULL_MASK, xb[CL * p0 / L], xl, L);
                nzb = vb != 0.0;
                if (nzb) vb = div_by_rcp(vb, piv.y, piv.x);
            }
            if (l == xl) {
                xa[CL * p0 / L] = va;
                if (ORD) xb[CL * p0 / L] = vb;
            }
#pragma unroll
            for (int t = 0; t < XN; ++t) {
                if (L * t > CL * p0 + CL - 1) continue;
                if (l + L * t < k) {
                    const double q = U[at[t].x + B.chunk(at[t], s) + p0];
                    if (nza) xa[t] = __dsub_rn(xa[t], __dmul_rn(va, q));
                    if (ORD && nzb) xb[t] = __dsub_rn(xb[t], __dmul_rn(vb, q));
                }
            }
        }
    }
    __syncwarp();
    return fail;
}

// ---------------------------------------------------------------------------
// The kernel: nodes to systems to outputs.

// Doubles of shared memory of a block's systems.
template <typename T>
__host__ __device__ constexpr int tile_smem(int warps) {
    return (warps * T::WARP + 1) & ~1;
}

// A group's node: rows l + L t of its system.
template <typename T>
struct TileNode {
    int node, n;
    int cell[T::XN];
    float dv[T::XN];  // cont: value - mean (float, combiner.h:18-22)
    int code[T::XN];  // IK: category code
    double b[T::XN];  // C(x_row - x0)
};

// The node's neighbour count and cells (node < 0: no node, an empty system).
template <typename T>
__device__ __forceinline__ void tile_fetch(const DevJob &J, const DevPlan &P, TileNode<T> &d, int node, int l) {
    d.node = node;
    d.n = 0;
#pragma unroll
    for (int t = 0; t < T::XN; ++t) d.cell[t] = 0;
    if (node < 0) return;
    d.n = J.nbcount[node];
    const int *lst = J.nb + (long long)node * P.nmax;
#pragma unroll
    for (int t = 0; t < T::XN; ++t)
        if (l + T::L * t < P.nmax) d.cell[t] = lst[l + T::L * t];
}

template <typename T>
__device__ __forceinline__ void tile_load(const DevJob &J, const DevPlan &P, double *U, TileNode<T> &d, int l) {
    int x0 = 0, y0 = 0, z0 = 0;
    if (d.node >= 0) node_xyz(J, d.node, x0, y0, z0);
#pragma unroll
    for (int t = 0; t < T::XN; ++t) {
        const int row = l + T::L * t;
        int2 o = make_int2(0, 0);
        d.dv[t] = 0.f;
        d.code[t] = -1;
        d.b[t] = 0.0;
        if (row < d.n) {
            const int cell = d.cell[t];
            int qx, qy, qz;
            node_xyz(J, cell, qx, qy, qz);
            qx -= x0;
            qy -= y0;
            qz -= z0;
            o.x = P.pk.pack(qx, qy, qz);
            o.y = qz * P.syx + qy * P.sx + qx;
            if (is_cont(J.kind)) {
                const float m = J.kind == 1 ? J.sk_mean_f : (J.kind == 2 ? J.mean[cell] : 0.f);
                d.dv[t] = __fsub_rn(J.values[cell], m);
            } else {
                d.code[t] = J.codes[cell];
            }
            d.b[t] = cov_lin(P, qx, qy, qz, o.y, J.err);
        }
        if (row < T::NC) reinterpret_cast<int2 *>(U + T::NBAT)[row] = o;
    }
    __syncwarp();
}

// init + t_0 + t_1 + ... + t_{n-1} in row order (row l + L t of the group
// holds term[t]), the same on every lane of the group.
template <typename T>
__device__ __forceinline__ float tile_fsum(double *vd, float init, const float (&term)[T::XN], int n, int nw, int l) {
    float *buf = reinterpret_cast<float *>(vd);
#pragma unroll
    for (int t = 0; t < T::XN; ++t)
        if (l + T::L * t < T::NC) buf[l + T::L * t] = term[t];
    __syncwarp();
    float r = init;
    const float4 *b4 = reinterpret_cast<const float4 *>(buf);
    for (int q = 0; 4 * q < nw; ++q) {
        const float4 v = b4[q];
        if (4 * q < n) r = __fadd_rn(r, v.x);
        if (4 * q + 1 < n) r = __fadd_rn(r, v.y);
        if (4 * q + 2 < n) r = __fadd_rn(r, v.z);
        if (4 * q + 3 < n) r = __fadd_rn(r, v.w);
    }
    __syncwarp();
    return r;
}
template <typename T>
__device__ __forceinline__ double tile_dsum(double *vd, double init, const double (&term)[T::XN], int n, int nw, int l) {
#pragma unroll
    for (int t = 0; t < T::XN; ++t)
        if (l + T::L * t < T::NC) vd[l + T::L * t] = term[t];
    __syncwarp();
    double r = init;
    const double2 *b2 = reinterpret_cast<const double2 *>(vd);
    for (int q = 0; 2 * q < nw; ++q) {
        const double2 v = b2[q];
        if (2 * q < n) r = __dadd_rn(r, v.x);
        if (2 * q + 1 < n) r = __dadd_rn(r, v.y);
    }
    __syncwarp();
    return r;
}

// Outputs of the group's system, as write_outputs.
template <typename T>
__device__ __forceinline__ void tile_outputs(const DevJob &J, const DevPlan &P, double *vd, const TileNode<T> &d,
                                             int nw, int l, int status, const double (&w)[T::XN], double variance) {
    const int node = d.node, n = d.n;
    const bool success = status == ST_SUCCESS, lead = l == 0 && node >= 0;
    const long long slot = (long long)node * J.status_stride + J.status_offset;
    if (J.weights && node >= 0) {
#pragma unroll
        for (int t = 0; t < T::XN; ++t)
            if (l + T::L * t < n) J.weights[slot * P.nmax + l + T::L * t] = w[t];
    }
    if (lead) {
        if (J.variance) J.variance[slot] = success ? variance : -1.0;
        J.status[slot] = (int8_t)status;
    }
    if (is_cont(J.kind)) {
        float term[T::XN];
#pragma unroll
        for (int t = 0; t < T::XN; ++t) term[t] = __double2float_rn(__dmul_rn(w[t], (double)d.dv[t]));
        const float m0 = J.kind == 1 ? J.sk_mean_f : (J.kind == 2 && node >= 0 ? J.mean[node] : 0.f);
        const float res = tile_fsum<T>(vd, m0, term, n, nw, l);
        if (lead) {
            if (success || J.kind != 0) {
                J.out_values[node] = success ? res : m0;
                J.out_mask[node] = 1;
            } else {
                J.untouched[atomicAdd(J.n_untouched, 1)] = node;
            }
        }
    } else if (J.kind == 3) {
        int best = 0;
        double best_p = 0;
        for (int k = J.k0; k < J.k1; ++k) {
            const float pk = J.pk[k];
            float term[T::XN];
#pragma unroll
            for (int t = 0; t < T::XN; ++t)
                term[t] = __double2float_rn(__dmul_rn(w[t], (double)__fsub_rn(d.code[t] == k ? 1.f : 0.f, pk)));
            const float sum = tile_fsum<T>(vd, pk, term, n, nw, l);
            const float prob = success ? sum : pk;
            if (lead) J.probs[(long long)node * J.K + k] = prob;
            if (k == J.k0 || (double)prob > best_p) {
                best_p = prob;
                best = k;
            }
        }
        if (J.k0 == 0 && J.k1 == J.K && lead) {
            J.out_codes[node] = (uint8_t)best;
            J.out_mask[node] = 1;
        }
    } else {
        const float m = J.median_m;
        double term[T::XN];
#pragma unroll
        for (int t = 0; t < T::XN; ++t) term[t] = __dmul_rn(w[t], (double)__fsub_rn(d.code[t] == 1 ? 1.f : 0.f, m));
        const double sum = tile_dsum<T>(vd, (double)m, term, n, nw, l);
        const double prob = success ? sum : (double)m;
        if (lead) {
            J.probs[node] = (float)prob;
            J.out_codes[node] = ((float)prob <= 0.5f) ? 0 : 1;
            J.out_mask[node] = 1;
        }
    }
}

// Solves the warp's loaded systems (d.node < 0: none for the group; nw: the
// largest neighbour count): the group's weights and, when asked for, its kriging
// variance.  Returns the group's status.
template <typename T>
__device__ __forceinline__ int tile_krige(const DevJob &J, const DevPlan &P, double *U, const TileTables<T> &B,
                                          TileNode<T> &d, int nw, int l, bool want_variance, double (&w)[T::XN],
                                          double &variance) {
    const int n = d.n;
    const bool ordinary = J.kind == 0;
    int status = n > 0 ? ST_SUCCESS : ST_NO_NEIGHBOURS;
#pragma unroll
    for (int t = 0; t < T::XN; ++t) w[t] = 0.0;
    if (nw <= 0) return status;
    double xb[T::XN];
#pragma unroll
    for (int t = 0; t < T::XN; ++t) {
        w[t] = d.b[t];
        xb[t] = l + T::L * t < n ? 1.0 : 0.0;
    }
    const bool singular = ordinary ? tile_solve<T, true>(J, P, U, B, n, nw, l, w, xb)
                                   : tile_solve<T, false>(J, P, U, B, n, nw, l, w, xb);
    if (n > 0 && singular) status = ST_SINGULAR;
    if (ordinary) {
        const double ssk = tile_dsum<T>(U, 0.0, w, n, nw, l);
        const double son = tile_dsum<T>(U, 0.0, xb, n, nw, l);
        const double mu = __ddiv_rn(__dsub_rn(ssk, 1.0), son);
#pragma unroll
        for (int t = 0; t < T::XN; ++t) w[t] = __dsub_rn(w[t], __dmul_rn(mu, xb[t]));
    }
    if (status != ST_SUCCESS) {
#pragma unroll
        for (int t = 0; t < T::XN; ++t) w[t] = 0.0;
    }
    if (want_variance) {
        // c0 - p_0 - p_1 - ... (my_kriging_weights.h): subtracting p is adding -p
        double p[T::XN];
#pragma unroll
        for (int t = 0; t < T::XN; ++t) p[t] = -__dmul_rn(w[t], d.b[t]);
        variance = tile_dsum<T>(U, P.c0, p, n, nw, l);
        if (ordinary) {
            double last = 0.0;
            const int at = n > 0 ? n - 1 : 0;
#pragma unroll
            for (int t = 0; t < T::XN; ++t) {
                const double q = __shfl_sync(FULL_MASK, w[t], at % T::L, T::L);
                if (at / T::L == t) last = q;
            }
            variance = __dsub_rn(variance, last);
        }
    }
    return status;
}

// The warp's systems and their outputs; returns the number of systems solved
// (on every lane).
template <typename T>
__device__ __forceinline__ int tile_systems(const DevJob &J, const DevPlan &P, double *U, const TileTables<T> &B,
                                            TileNode<T> &d, int l) {
    const int nw = __reduce_max_sync(FULL_MASK, d.n);
    double w[T::XN], variance = -1.0;
    if (nw > 0) tile_load<T>(J, P, U, d, l);
    const int status = tile_krige<T>(J, P, U, B, d, nw, l, J.variance != nullptr, w, variance);
    tile_outputs<T>(J, P, U, d, nw, l, status, w, variance);
    __syncwarp();
    return __popc(__ballot_sync(FULL_MASK, l == 0 && d.n > 0));
}

// Every node of the job.  Warps take up to 32 consecutive nodes at a time from
// the per-job counter, copy the informed ones' values, and solve the others
// T::G at a time, across chunks; the next systems' lists are read while the
// current ones are solved.
template <typename T, int WARPS, int MINB>
__global__ void __launch_bounds__(WARPS * 32, MINB) k_solve_tile(DevJob J, DevPlan P) {
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    double *systems = reinterpret_cast<double *>(dyn_smem);
    TileTables<T> &B = *reinterpret_cast<TileTables<T> *>(systems + tile_smem<T>(WARPS));
    B.fill(threadIdx.x, WARPS * 32);
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int group = lane / T::L, l = lane % T::L;
    double *U = systems + warp * T::WARP + group * T::STRIDE;
    // small jobs: fewer nodes a chunk, down to one per group, so that every
    // warp gets some
    const int csize = max(T::G, chunk_nodes(J, 32, WARPS));
    unsigned long long solved = 0;
    unsigned m = 0;  // the chunk's nodes still to solve (bit b: node base + b)
    int base = 0;
    bool more = true;
    // the group's next node, or -1
    auto take = [&]() {
        int node = -1;
#pragma unroll 1
        for (int g = 0; g < T::G; ++g) {
            while (more && !m) {
                int c = 0;
                if (lane == 0) c = atomicAdd(J.node_next, csize);
                base = __shfl_sync(FULL_MASK, c, 0);
                more = chunk_first(base, J.size) < J.size;
                const int i = (int)((unsigned)base + (unsigned)lane);
                bool solve = more && chunk_has(base, lane, csize, J.size);
                if (solve && is_cont(J.kind) && J.mask[i] != 0) {
                    J.out_values[i] = J.values[i];
                    J.out_mask[i] = 1;
                    J.status[(long long)i * J.status_stride + J.status_offset] = ST_NOT_KRIGED;
                    solve = false;
                }
                m = __ballot_sync(FULL_MASK, solve);
            }
            if (m) {
                if (g == group) node = base + __ffs(m) - 1;
                m &= m - 1;
            }
        }
        return node;
    };
    TileNode<T> next;
    tile_fetch<T>(J, P, next, take(), l);
    while (__any_sync(FULL_MASK, next.node >= 0)) {
        TileNode<T> cur = next;
        tile_fetch<T>(J, P, next, take(), l);
        solved += tile_systems<T>(J, P, U, B, cur, l);
    }
    if (lane == 0 && solved) atomicAdd(J.n_fp64, solved);
}

// The next systems of the round's solve list, T::G at a time: the group's node,
// its list (list `which` of the `lists` a window slot has) and path rank;
// false once the list is used up.
template <typename T>
__device__ __forceinline__ bool sgs_next_systems(const SgsState &G, const int *win, int count, int stride, int lists,
                                                 int which, int lane, TileNode<T> &d, int &rank) {
    const int group = lane / T::L, l = lane % T::L;
    int first = 0;
    if (lane == 0) first = (int)atomicAdd(&G.ctl->solve_cursor, (unsigned)T::G);
    first = __shfl_sync(FULL_MASK, first, 0);
    if (first >= count) return false;
    d.node = -1;
    d.n = 0;
    rank = 0;
#pragma unroll
    for (int t = 0; t < T::XN; ++t) d.cell[t] = 0;
    if (first + group < count) {
        const int slot = G.solvelist[first + group];
        rank = win[slot];
        d.node = G.nodes[rank];
        const long long at = (long long)slot * lists + which;
        d.n = G.counts[at];
        const int *lst = G.lists + at * stride;
#pragma unroll
        for (int t = 0; t < T::XN; ++t)
            if (l + T::L * t < d.n) d.cell[t] = lst[l + T::L * t];
    }
    return true;
}

// The systems of a simulation round's finished searches (G.solvelist, in any
// order): the lists lie by window slot, and the simulated value is xp
// sqrt(variance) + estimate, or xp where the kriging fails
// (sequential_simulation.h:106-110, gaussian_distribution.h:49-66).
template <typename T, int WARPS, int MINB>
__global__ void __launch_bounds__(WARPS * 32, MINB) k_sgs_solve(DevJob J, DevPlan P, SgsState G, int cur) {
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    double *systems = reinterpret_cast<double *>(dyn_smem);
    TileTables<T> &B = *reinterpret_cast<TileTables<T> *>(systems + tile_smem<T>(WARPS));
    B.fill(threadIdx.x, WARPS * 32);
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int group = lane / T::L, l = lane % T::L;
    double *U = systems + warp * T::WARP + group * T::STRIDE;
    const int count = G.ctl->nsolve;
    const int *win = cur ? G.win1 : G.win0;
    TileNode<T> d;
    int rank;
    while (sgs_next_systems<T>(G, win, count, P.nmax, 1, 0, lane, d, rank)) {
        const bool mine = d.node >= 0;
        const int nw = __reduce_max_sync(FULL_MASK, d.n);
        double w[T::XN], variance = 0.0;
        if (nw > 0) tile_load<T>(J, P, U, d, l);
        const int status = tile_krige<T>(J, P, U, B, d, nw, l, true, w, variance);
        float est = 0.f;
        if (nw > 0) {
            float term[T::XN];
#pragma unroll
            for (int t = 0; t < T::XN; ++t) term[t] = __double2float_rn(__dmul_rn(w[t], (double)d.dv[t]));
            const float m0 = J.kind == 1 ? J.sk_mean_f : (J.kind == 2 && mine ? J.mean[d.node] : 0.f);
            est = tile_fsum<T>(U, m0, term, d.n, nw, l);
        }
        if (mine && l == 0) {
            const double xp = G.xp[rank];
            const double value = status == ST_SUCCESS ? __dadd_rn(__dmul_rn(xp, __dsqrt_rn(variance)), (double)est)
                                                      : __dadd_rn(__dmul_rn(xp, 1.0), 0.0);
            J.sim_values[d.node] = __double2float_rn(value);
            J.sim_mask[d.node] = 1;
        }
        __syncwarp();
    }
}

// The same for indicator simulation: the system of categories [k0, k1), which
// share a covariance model and search, solved once; per category the
// probability m_c + sum w_i (ind_i - m_i) accumulated in double
// (kriging_interpolation.h:228-265), the category's mean where the kriging
// fails.  Two categories krige category 0 only and take 1 - p for the other.
template <typename T, int WARPS, int MINB>
__global__ void __launch_bounds__(WARPS * 32, MINB) k_sis_solve(DevJob J, DevPlan P, SgsState G, int cur, int stride,
                                                                int lists, int which, int k0, int k1) {
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    double *systems = reinterpret_cast<double *>(dyn_smem);
    TileTables<T> &B = *reinterpret_cast<TileTables<T> *>(systems + tile_smem<T>(WARPS));
    B.fill(threadIdx.x, WARPS * 32);
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int group = lane / T::L, l = lane % T::L;
    double *U = systems + warp * T::WARP + group * T::STRIDE;
    const int count = G.ctl->nsolve;
    const int *win = cur ? G.win1 : G.win0;
    TileNode<T> d;
    int rank;
    while (sgs_next_systems<T>(G, win, count, stride, lists, which, lane, d, rank)) {
        const bool mine = d.node >= 0;
        const int nw = __reduce_max_sync(FULL_MASK, d.n);
        double w[T::XN], variance = 0.0;
        if (nw > 0) tile_load<T>(J, P, U, d, l);
        const int status = tile_krige<T>(J, P, U, B, d, nw, l, false, w, variance);
        for (int k = k0; k < k1; ++k) {
            const float mc = mine ? sis_mean(J, k, d.node) : 0.f;
            double prob = (double)mc;
            if (nw > 0) {
                double term[T::XN];
#pragma unroll
                for (int t = 0; t < T::XN; ++t) {
                    const float m = l + T::L * t < d.n ? sis_mean(J, k, d.cell[t]) : 0.f;
                    term[t] = __dmul_rn(w[t], (double)__fsub_rn(d.code[t] == k ? 1.f : 0.f, m));
                }
                const double sum = tile_dsum<T>(U, (double)mc, term, d.n, nw, l);
                if (status == ST_SUCCESS) prob = sum;
            }
            if (mine && l == 0) {
                float *probs = J.probs + (long long)d.node * J.K;
                probs[k] = __double2float_rn(prob);
                if (J.K == 2) probs[1] = __double2float_rn(__dsub_rn(1.0, prob));
            }
        }
        __syncwarp();
    }
}

template <typename T, int WARPS, int MINB>
static void launch_sis_solve(const DevJob &J, const DevPlan &P, const SgsState &G, int cur, int stride, int lists,
                             int which, int k0, int k1, cudaStream_t s) {
    constexpr size_t smem = sizeof(double) * tile_smem<T>(WARPS) + sizeof(TileTables<T>);
    const long long g = persistent_grid((const void *)k_sis_solve<T, WARPS, MINB>, WARPS * 32, smem, 0, 1LL << 30);
    k_sis_solve<T, WARPS, MINB><<<(unsigned)g, WARPS * 32, smem, s>>>(J, P, G, cur, stride, lists, which, k0, k1);
}

template <typename T, int WARPS, int MINB>
static void launch_sgs_solve(const DevJob &J, const DevPlan &P, const SgsState &G, int cur, cudaStream_t s) {
    constexpr size_t smem = sizeof(double) * tile_smem<T>(WARPS) + sizeof(TileTables<T>);
    const long long g = persistent_grid((const void *)k_sgs_solve<T, WARPS, MINB>, WARPS * 32, smem, 0, 1LL << 30);
    k_sgs_solve<T, WARPS, MINB><<<(unsigned)g, WARPS * 32, smem, s>>>(J, P, G, cur);
}

template <typename T, int WARPS, int MINB>
static void launch_tile(const DevJob &J, const DevPlan &P, cudaStream_t s, int blocks_per_sm) {
    constexpr size_t smem = sizeof(double) * tile_smem<T>(WARPS) + sizeof(TileTables<T>);
    const long long units = (J.size + WARPS * T::G - 1) / (WARPS * T::G);
    const long long g = persistent_grid((const void *)k_solve_tile<T, WARPS, MINB>, WARPS * 32, smem, blocks_per_sm, units);
    k_solve_tile<T, WARPS, MINB><<<(unsigned)g, WARPS * 32, smem, s>>>(J, P);
}

}  // namespace hpgl_b200
