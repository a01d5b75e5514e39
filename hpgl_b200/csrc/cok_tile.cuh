// Colocated cokriging systems on lane tiles: gauss_solve (gauss_solver.cpp:
// 5-63) in the reference's operation order, several systems per warp.
//
// The elimination is not symmetric in its roundings (a(r,k) -= a(r,i) *
// (a(i,k) / a(i,i))), so the whole square is updated, in place.  With one
// system a warp and a row per lane each product read its pivot entry and its
// own entry from shared memory and wrote it back; here a system takes L = CL x
// RL lanes, lane (r, c) holds rows r mod RL and columns c mod CL in
// registers, and a step exchanges one row and one column through shared
// memory.  Products with rows and columns of later blocks wait until the next
// pivot's chain runs, as in the kriging solves.  The pivot order is the
// natural one whenever no diagonal entry vanishes; a system where one does
// (or where a pivot leaves recip's range) is marked, and the one-system-a-warp
// kernel solves it with its search for a pivot row.
//
// Measured on 161x119x47 (0.88 M systems of 24 neighbours): 4.5 ms where one
// system a warp took 13.7; the pivot chain's latency and the exchange through
// shared memory bound it, 7 warps an SM for their registers.
#pragma once
#include "device_common.cuh"
#include "tile_geom.h"

namespace hpgl_b200 {

constexpr int8_t COK_REDO = 3;  // status of a marked node until it is solved

// RN(1 / a) without a branch for 2^-900 <= |a| < 2^900 (false otherwise):
// Newton's iteration from the hardware's approximate reciprocal, the last
// two steps Markstein's (IBM J. Res. Dev. 34(1), 1990), the first of them
// rounded away from zero so that a significand of ones rounds correctly too.
__device__ __forceinline__ bool recip(double a, double &rcp) {
    const double m = fabs(a);
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(m));
    y = __fma_rn(__fma_rn(-m, y, 1.0), y, y);
    y = __fma_ru(__fma_rn(-m, y, 1.0), y, y);
    y = __fma_rn(__fma_rn(-m, y, 1.0), y, y);
    rcp = copysign(y, a);
    return (unsigned)__double2hiint(m) - 0x07b00000u < 0x70800000u;  // exponents 123 .. 1922
}

// The group's system in shared memory (row-major tiles, at()): covariances,
// the secondary's row and column n, B; the identity beyond.  x: the lane's
// neighbours' values (rows l + L t).
template <typename T>
__device__ __forceinline__ void cok_build(const DevJob &J, const DevPlan &P, double *S, int node, int n, int l,
                                          float (&x)[T::XN]) {
    int2 *nb = reinterpret_cast<int2 *>(S + T::COL);
    int2 own[T::XN];
    double bv[T::XN], cr[T::XN];
    int x0 = 0, y0 = 0, z0 = 0;
    if (node >= 0) node_xyz(J, node, x0, y0, z0);
#pragma unroll
    for (int t = 0; t < T::XN; ++t) {
        const int row = l + T::L * t;
        int2 o = make_int2(0, 0);
        x[t] = 0.f;
        bv[t] = cr[t] = 0.0;
        if (row < n) {
            const int cell = J.nb[(long long)node * P.nmax + row];
            int qx, qy, qz;
            node_xyz(J, cell, qx, qy, qz);
            qx -= x0;
            qy -= y0;
            qz -= z0;
            o.x = P.pk.pack(qx, qy, qz);
            o.y = qz * P.syx + qy * P.sx + qx;
            x[t] = J.values[cell];
            // primary_cov(x_r, center); cross_cov(center, x_r) = coef C_x(center - x_r)
            bv[t] = cov_lin(P, qx, qy, qz, o.y, J.err);
            double cx = 0.0;
            if (cov_in_range(P, qx, qy, qz)) cx = __ldg(J.cross_table + abs(o.y));
            cr[t] = __dmul_rn(J.cok_coef, cx);
        }
        own[t] = o;
        if (row < T::NN) nb[row] = o;
    }
    __syncwarp();
    // every pair of neighbours once, a batch of a lane's gathers in flight
    constexpr int PAIRS = T::XN * (T::NN / 2), BATCH = 16;
    bool out = false;
#pragma unroll
    for (int e0 = 0; e0 < PAIRS; e0 += BATCH) {
        double v[BATCH];
#pragma unroll
        for (int e = 0; e < BATCH; ++e) {
            if (e0 + e >= PAIRS) continue;
            const int t = (e0 + e) % T::XN, d = (e0 + e) / T::XN + 1;
            const int i = l + T::L * t;
            int k = i + d;
            if (k >= T::NN) k -= T::NN;
            v[e] = 0.0;
            if (i < n && k < n && (d < T::NN / 2 || i < T::NN / 2)) {
                const int2 q = nb[k];
                const bool in = P.pk.in_range((int)((unsigned)own[t].x - (unsigned)q.x));
                if (in) v[e] = __ldg(P.table + abs(own[t].y - q.y));
                out |= !in;
            }
        }
#pragma unroll
        for (int e = 0; e < BATCH; ++e) {
            if (e0 + e >= PAIRS) continue;
            const int t = (e0 + e) % T::XN, d = (e0 + e) / T::XN + 1;
            const int i = l + T::L * t;
            int k = i + d;
            if (k >= T::NN) k -= T::NN;
            if (i < T::NN && (d < T::NN / 2 || i < T::NN / 2)) {
                S[T::at(i, k)] = v[e];
                S[T::at(k, i)] = v[e];
            }
        }
    }
    if (out && !P.truncated) atomicOr(J.err, DERR_TABLE_RANGE);
    // columns NN and beyond (and rows from NN on): zero, then row and column n
    for (int e = l; e < T::NR * (T::NC - T::NN); e += T::L) S[T::at(e % T::NR, T::NN + e / T::NR)] = 0.0;
    for (int e = l; e < (T::NR - T::NN) * T::NN; e += T::L) S[T::at(T::NN + e / T::NN, e % T::NN)] = 0.0;
    __syncwarp();
    const double c0 = __ldg(P.table);
    for (int i = l; i < T::NR; i += T::L) S[T::at(i, i)] = i < n ? c0 : i == n ? J.cok_svar : 1.0;
#pragma unroll
    for (int t = 0; t < T::XN; ++t) {
        const int row = l + T::L * t;
        if (row < n) {
            S[T::at(row, n)] = cr[t];
            S[T::at(n, row)] = cr[t];
            S[T::at(row, T::BCOL)] = bv[t];
        }
    }
    if (l == 0) S[T::at(n, T::BCOL)] = __dmul_rn(J.cok_coef, __ldg(J.cross_table));
    __syncwarp();
}

// Eliminates and back-substitutes the warp's systems (ms unknowns, mw the
// most in the warp); x[t]: unknown l + L t.  Returns whether the natural pivot
// order held.
template <typename T>
__device__ __forceinline__ bool cok_solve(double *S, int ms, int mw, int l, double (&x)[T::XN]) {
    constexpr int NBR = T::NBR, NBC = T::NBC, CL = T::CL, RL = T::RL, L = T::L, H = T::H;
    const int r = l / CL, c = l % CL;
    double t[NBR][NBC], u[NBC + 1], w[NBR + 1];
#pragma unroll
    for (int a = 0; a < NBR; ++a) {
        const double2 *p = reinterpret_cast<const double2 *>(S + (RL * a + r) * T::RS + T::off(c));
#pragma unroll
        for (int b = 0; b < NBC; b += 2) {
            const double2 q = p[b / 2];
            t[a][b] = q.x;
            if (b + 1 < NBC) t[a][b + 1] = q.y;
        }
        w[a] = 0.0;
    }
#pragma unroll
    for (int b = 0; b < NBC; ++b) u[b] = 0.0;
    __syncwarp();
    bool ok = true;
#pragma unroll
    for (int p0 = 0; p0 < NBC; ++p0) {
        if (CL * p0 >= mw) break;
#pragma unroll
        for (int h0 = 0; h0 < H; ++h0) {
            if (p0 * H + h0 >= NBR) continue;
#pragma unroll 1
            for (int rr = 0; rr < RL; ++rr) {
                const int s = h0 * RL + rr, i = CL * p0 + s;
                double *row = S + i * T::RS + T::off(c);
                double *col = S + T::COL + (i & 1) * (RL * T::CR) + r * T::CR;
                const double coef = __shfl_sync(FULL_MASK, t[p0 * H + h0][p0], rr * CL + s, L);
                // the products that waited
#pragma unroll
                for (int a = (p0 + 1) * H; a < NBR; ++a)
#pragma unroll
                    for (int b = p0 + 1; b < NBC; ++b) t[a][b] = __dsub_rn(t[a][b], __dmul_rn(w[a], u[b]));
                double y;
                ok &= recip(coef, y);
                if (r == rr) {
                    // the normalised pivot row
#pragma unroll
                    for (int b = p0 & ~1; b < NBC; b += 2) {
                        double2 q;
                        q.x = b >= p0 ? div_by_rcp(t[p0 * H + h0][b], coef, y) : 0.0;
                        q.y = b + 1 < NBC ? div_by_rcp(t[p0 * H + h0][b + 1], coef, y) : 0.0;
                        *reinterpret_cast<double2 *>(row + b) = q;
                    }
                }
                if (c == s) {
#pragma unroll
                    for (int a = p0 * H & ~1; a < NBR; a += 2)
                        *reinterpret_cast<double2 *>(col + a) = make_double2(t[a][p0], a + 1 < NBR ? t[a + 1][p0] : 0.0);
                }
                __syncwarp();
#pragma unroll
                for (int b = p0 & ~1; b < NBC; b += 2) {
                    const double2 q = *reinterpret_cast<const double2 *>(row + b);
                    u[b] = q.x;
                    u[b + 1] = q.y;
                }
#pragma unroll
                for (int a = p0 * H & ~1; a < NBR; a += 2) {
                    const double2 q = *reinterpret_cast<const double2 *>(col + a);
                    w[a] = q.x;
                    w[a + 1] = q.y;
                }
                // the block's own rows and columns take them at once
#pragma unroll
                for (int a = p0 * H; a < NBR && a < (p0 + 1) * H; ++a)
#pragma unroll
                    for (int b = p0; b < NBC; ++b) t[a][b] = __dsub_rn(t[a][b], __dmul_rn(w[a], u[b]));
#pragma unroll
                for (int a = (p0 + 1) * H; a < NBR; ++a) t[a][p0] = __dsub_rn(t[a][p0], __dmul_rn(w[a], u[p0]));
            }
        }
        // the next block's rows and columns take the last row's products now
        if (p0 + 1 < NBC) {
#pragma unroll
            for (int a = (p0 + 1) * H; a < NBR && a < (p0 + 2) * H; ++a)
#pragma unroll
                for (int b = p0 + 1; b < NBC; ++b) t[a][b] = __dsub_rn(t[a][b], __dmul_rn(w[a], u[b]));
#pragma unroll
            for (int a = (p0 + 2) * H; a < NBR; ++a)
                t[a][p0 + 1] = __dsub_rn(t[a][p0 + 1], __dmul_rn(w[a], u[p0 + 1]));
        }
    }
    // X[i] = B[i] - sum_{j > i, j descending} A[i][j] X[j]
#pragma unroll
    for (int q = 0; q < T::XN; ++q) x[q] = l + L * q < ms ? S[T::at(l + L * q, T::BCOL)] : 0.0;
#pragma unroll
    for (int tj = T::XN - 1; tj >= 0; --tj) {
#pragma unroll 1
        for (int lj = L - 1; lj >= 0; --lj) {
            const int j = lj + L * tj;
            if (j >= mw || j == 0) continue;
            const double xj = __shfl_sync(FULL_MASK, x[tj], lj, L);
#pragma unroll
            for (int q = 0; q <= tj; ++q)
                if (l + L * q < j && j < ms)
                    x[q] = __dsub_rn(x[q], __dmul_rn(S[(l + L * q) * T::RS + T::off(j % CL) + j / CL], xj));
        }
    }
    return ok;
}

// Every uninformed node's system.  Warps take up to 32 consecutive nodes at a
// time from the per-job counter and solve them T::G at a time, across chunks.
template <typename T, int WARPS, int MINB>
__global__ void __launch_bounds__(WARPS * 32, MINB) k_cok_tile(DevJob J, DevPlan P) {
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int group = lane / T::L, l = lane % T::L;
    double *S = reinterpret_cast<double *>(dyn_smem) + (size_t)(warp * T::G + group) * T::SIZE;
    const float m1 = J.cok_m1, m2 = J.cok_m2;
    const int csize = max(T::G, chunk_nodes(J, 32, WARPS));
    unsigned long long solved = 0;
    unsigned m = 0;
    int base = 0;
    bool more = true;
    while (true) {
        int node = -1;
#pragma unroll 1
        for (int g = 0; g < T::G; ++g) {
            while (more && !m) {
                int k = 0;
                if (lane == 0) k = atomicAdd(J.node_next, csize);
                base = __shfl_sync(FULL_MASK, k, 0);
                more = chunk_first(base, J.size) < J.size;
                const int i = (int)((unsigned)base + (unsigned)lane);
                bool solve = more && chunk_has(base, lane, csize, J.size);
                if (solve && J.mask[i]) {
                    // informed primary: copied (set_at, simple_cokriging_markI.cpp:245-248)
                    J.out_values[i] = J.values[i];
                    J.out_mask[i] = 1;
                    J.status[i] = ST_NOT_KRIGED;
                    solve = false;
                }
                m = __ballot_sync(FULL_MASK, solve);
            }
            if (m) {
                if (g == group) node = base + __ffs(m) - 1;
                m &= m - 1;
            }
        }
        if (!__any_sync(FULL_MASK, node >= 0)) break;
        const int n = node >= 0 ? J.nbcount[node] : 0;
        const float sv = node >= 0 ? (J.smask[node] ? J.svalues[node] : m2) : 0.f;
        const int nw = __reduce_max_sync(FULL_MASK, n);
        float result = __fsub_rn(__fadd_rn(m1, sv), m2);  // failure estimate
        int status = ST_NO_NEIGHBOURS;
        double w[T::XN];
        if (nw > 0) {
            float v[T::XN];
            cok_build<T>(J, P, S, node, n, l, v);
            const bool ok = cok_solve<T>(S, n + 1, nw + 1, l, w);
            if (n > 0) status = ok ? ST_SUCCESS : COK_REDO;
            // combine (simple_cokriging_markI.cpp:84-105): float result, each
            // step widened to double and rounded back
            double *p = S;
            __syncwarp();
#pragma unroll
            for (int t = 0; t < T::XN; ++t) {
                const int i = l + T::L * t;
                if (i < n) p[i] = __dmul_rn((double)__fsub_rn(v[t], m1), w[t]);
                if (i == n) p[i] = __dmul_rn(w[t], (double)__fsub_rn(sv, m2));
            }
            __syncwarp();
            float res = m1;
            for (int i = 0; i <= nw; ++i) {
                const double q = p[i];
                if (i <= n) res = __double2float_rn(__dadd_rn((double)res, q));
            }
            if (status == ST_SUCCESS) result = res;
            __syncwarp();
        }
        if (node >= 0) {
            if (l == 0) {
                J.out_values[node] = result;
                J.out_mask[node] = 1;
                J.status[node] = (int8_t)status;
            }
            if (J.weights && status == ST_SUCCESS) {
                double *dst = J.weights + (long long)node * (P.nmax + 1);
#pragma unroll
                for (int t = 0; t < T::XN; ++t)
                    if (l + T::L * t <= n) dst[l + T::L * t] = w[t];
            }
        }
        solved += __popc(__ballot_sync(FULL_MASK, l == 0 && status == ST_SUCCESS));
    }
    if (lane == 0 && solved) atomicAdd(J.n_fp64, solved);
}

}  // namespace hpgl_b200
