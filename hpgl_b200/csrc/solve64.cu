// Per-node solves for systems of 33 to 64 neighbours, FP64 in the reference's
// exact operation order (my_kriging_weights.h:26-255 over LAPACK DPOTF2 /
// DPOTRS).
//
//   k_solve_tile    (tile_solve.cuh) two systems a warp (above 56 neighbours
//                   one, on all its lanes), persistent over the grid's
//                   nodes: every kriging job's solve.
//   exact64_core    one system a warp, lane l owning rows and columns l and
//                   l + 32: sequential simulation, the fused search + solve
//                   kernel, and the jobs the tiled kernels do not take
//                   (k_solve_exact64).  The system and its factor live in a
//                   skewed packed upper triangle in shared memory: every lane
//                   reads its own columns as conflict-free 16-byte pairs while
//                   the column of the step is broadcast, and the forward
//                   substitution U^T y = b runs inside the factorisation (row
//                   j of U is final at step j, which is all the dot-product
//                   form of DTRSM needs).  The step loop is a plain runtime
//                   loop, so the kernel stays small for the instruction
//                   caches.
#include <algorithm>

#include "device_common.cuh"
#include "search_common.cuh"
#include "tile_solve.cuh"

namespace hpgl_b200 {

namespace {

constexpr int N64 = 64;

constexpr int WARPS64_BLOCK = 1;

// At most this many nodes a 64-row solve warp takes from the per-job counter at a time, and the
// taking itself (lane 0's atomic, broadcast).
constexpr int CHUNK64 = 16;
__device__ __forceinline__ int take_chunk64(const DevJob &J, int lane, int csize) {
    int c = 0;
    if (lane == 0) c = atomicAdd(J.node_next, csize);
    return __shfl_sync(FULL_MASK, c, 0);
}

// The factor lives in shared memory as a skewed packed upper triangle:
// column k starts at col_start(k), holds rows 0..k (padded to an even count)
// and col_start(k) = 2k (mod 16) doubles, so when every lane reads a 16-byte
// pair of its own column at the same row, the 32 addresses fall on 8
// different 16-byte bank groups, 4 each: conflict-free.  Column k is the
// matrix column A(., k) until its rows are overwritten, one per step, by the
// factor's row; its diagonal slot stays zero until step k.
// (col_start_c runs a loop: device code reads the starts from a table the
// kernels fill once per block.)
__host__ __device__ constexpr int col_start_c(int k) {
    int start = 0, end = 0;
    for (int c = 0; c <= k; ++c) {
        start = end;
        while ((start & 15) != ((2 * c) & 15)) ++start;
        end = start + ((c + 2) & ~1);
    }
    return start;
}
constexpr int U64_SIZE = col_start_c(N64 - 1) + N64;  // 2558 doubles
static_assert(col_start_c(3) == 22 && U64_SIZE == 2558, "skewed layout");

struct Exact64Smem {
    double U[U64_SIZE];
    int4 nb[N64];     // neighbour offsets from the node (x, y, z, table offset)
};

__device__ __noinline__ double dsqrt64(double a) { return __dsqrt_rn(a); }
__device__ __noinline__ double drcp64(double a) { return __drcp_rn(a); }

struct Node64 {
    int n;
    float dv[2];  // cont: value - mean (float, combiner.h:18-22)
    int code[2];  // IK: category code
    double b[2];  // C(x_row - x0)
};

__device__ __forceinline__ Node64 load_node64(const DevJob &J, const DevPlan &P, int4 *nb, const NodeFetch &f,
                                              int lane) {
    Node64 d;
    const int node = f.node;
    d.n = f.n;
    int x0, y0, z0;
    node_xyz(J, node, x0, y0, z0);
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int row = lane + 32 * r;
        d.dv[r] = 0.f;
        d.code[r] = -1;
        d.b[r] = 0.0;
        int4 o = make_int4(0, 0, 0, 0);
        if (row < d.n) {
            const int cell = r ? f.cell2 : f.cell;
            int qx, qy, qz;
            node_xyz(J, cell, qx, qy, qz);
            o.x = qx - x0;
            o.y = qy - y0;
            o.z = qz - z0;
            o.w = o.z * P.syx + o.y * P.sx + o.x;
            if (is_cont(J.kind)) {
                const float m = J.kind == 1 ? J.sk_mean_f : (J.kind == 2 ? J.mean[cell] : 0.f);
                d.dv[r] = __fsub_rn(J.values[cell], m);
            } else {
                d.code[r] = J.codes[cell];
            }
            d.b[r] = cov_lin(P, o.x, o.y, o.z, o.w, J.err);
        }
        nb[row] = o;
    }
    __syncwarp();
    return d;
}

// Value of row i (0..63) held as (v0 in lane i) / (v1 in lane i - 32).
template <typename T>
__device__ __forceinline__ T row_val(T v0, T v1, int i) {
    return i < 32 ? __shfl_sync(FULL_MASK, v0, i) : __shfl_sync(FULL_MASK, v1, i - 32);
}

// init + v_0 + v_1 + ... + v_{n-1} in row order (v_i held as v0 in lane i
// for i < 32, v1 in lane i - 32 above), float or double.
__device__ __forceinline__ float rows_fsum(float acc, float v0, float v1, int n) {
    const int n0 = n < 32 ? n : 32;
    for (int i = 0; i < n0; ++i) acc = __fadd_rn(acc, __shfl_sync(FULL_MASK, v0, i));
    for (int i = 32; i < n; ++i) acc = __fadd_rn(acc, __shfl_sync(FULL_MASK, v1, i - 32));
    return acc;
}
__device__ __forceinline__ double rows_dsum(double acc, double v0, double v1, int n) {
    const int n0 = n < 32 ? n : 32;
    for (int i = 0; i < n0; ++i) acc = __dadd_rn(acc, __shfl_sync(FULL_MASK, v0, i));
    for (int i = 32; i < n; ++i) acc = __dadd_rn(acc, __shfl_sync(FULL_MASK, v1, i - 32));
    return acc;
}

// Outputs of one solved (or failed) system, weights w0/w1 of rows lane and
// lane + 32; the same combination rules as the 32-neighbour kernels.
__device__ __forceinline__ void write_outputs64(const DevJob &J, const DevPlan &P, int node, int lane,
                                                const Node64 &d, int status, double w0, double w1,
                                                double variance) {
    const long long slot = (long long)node * J.status_stride + J.status_offset;
    const bool success = status == ST_SUCCESS;
    const int n = d.n;
    if (J.weights && n > 0) {
        if (lane < n) J.weights[slot * P.nmax + lane] = w0;
        if (lane + 32 < n) J.weights[slot * P.nmax + lane + 32] = w1;
    }
    if (J.variance && lane == 0) J.variance[slot] = success ? variance : -1.0;
    if (lane == 0) J.status[slot] = (int8_t)status;
    if (is_cont(J.kind)) {
        if (success) {
            // combine (combiner.h:9-24): float sum in neighbour order.
            const float t0 = __double2float_rn(__dmul_rn(w0, (double)d.dv[0]));
            const float t1 = __double2float_rn(__dmul_rn(w1, (double)d.dv[1]));
            float res = J.kind == 1 ? J.sk_mean_f : (J.kind == 2 ? J.mean[node] : 0.f);
            res = rows_fsum(res, t0, t1, n);
            if (lane == 0) {
                J.out_values[node] = res;
                J.out_mask[node] = 1;
            }
        } else if (lane == 0) {
            if (J.kind == 0) {
                const int pos = atomicAdd(J.n_untouched, 1);
                J.untouched[pos] = node;
            } else {
                J.out_values[node] = J.kind == 1 ? J.sk_mean_f : J.mean[node];
                J.out_mask[node] = 1;
            }
        }
    } else if (J.kind == 3) {
        int best = 0;
        double best_p = 0;
        for (int k = J.k0; k < J.k1; ++k) {
            const float pk = J.pk[k];
            float prob = pk;
            if (success) {
                const float t0 =
                    __double2float_rn(__dmul_rn(w0, (double)__fsub_rn(d.code[0] == k ? 1.f : 0.f, pk)));
                const float t1 =
                    __double2float_rn(__dmul_rn(w1, (double)__fsub_rn(d.code[1] == k ? 1.f : 0.f, pk)));
                prob = rows_fsum(prob, t0, t1, n);
            }
            if (lane == 0) J.probs[(long long)node * J.K + k] = prob;
            if (k == J.k0 || (double)prob > best_p) {
                best_p = prob;
                best = k;
            }
        }
        if (J.k0 == 0 && J.k1 == J.K && lane == 0) {
            J.out_codes[node] = (uint8_t)best;
            J.out_mask[node] = 1;
        }
    } else {
        const float m = J.median_m;
        double prob = (double)m;
        if (success) {
            const double t0 = __dmul_rn(w0, (double)__fsub_rn(d.code[0] == 1 ? 1.f : 0.f, m));
            const double t1 = __dmul_rn(w1, (double)__fsub_rn(d.code[1] == 1 ? 1.f : 0.f, m));
            prob = rows_dsum(prob, t0, t1, n);
        }
        if (lane == 0) {
            J.probs[node] = (float)prob;
            J.out_codes[node] = ((float)prob <= 0.5f) ? 0 : 1;
            J.out_mask[node] = 1;
        }
    }
}

__device__ __forceinline__ bool copy_informed64(const DevJob &J, const NodeFetch &f, int lane) {
    const int node = f.node;
    if (f.informed) {
        if (lane == 0) {
            J.out_values[node] = J.values[node];
            J.out_mask[node] = 1;
            J.status[(long long)node * J.status_stride + J.status_offset] = ST_NOT_KRIGED;
        }
        return true;
    }
    return false;
}

__device__ __forceinline__ double pair_cov64(const DevJob &J, const DevPlan &P, const int4 &a, const int4 &b) {
    // C(x_a - x_b) (my_kriging_weights.h:53, 160)
    return cov_lin(P, a.x - b.x, a.y - b.y, a.z - b.z, a.w - b.w, J.err);
}

// Build: the n(n-1)/2 entries A(i, k) = C(x_i - x_k), i < k, of the upper
// triangle into the skewed packed layout (my_kriging_weights.h:49-58; the
// tables are exactly symmetric, C(v) = C(-v) bit for bit, so either
// orientation gives the reference's value).  Lane l takes the pairs
// (r, r + d mod 64) of its rows r = l, l + 32 for d = 1..31, and (l, l + 32):
// every pair once, 63 a lane, 16 gathers in flight per trip.  Columns from n
// on are left as they are.
template <bool CORR>
__device__ __forceinline__ void build_packed(const DevJob &J, const DevPlan &P, double *U, const int4 *nb,
                                             const int *cs, int n, int lane, const double *sg) {
    const int4 own[2] = {nb[lane], nb[lane + 32]};
#pragma unroll 1
    for (int d0 = 1; d0 <= 32; d0 += 8) {
        double v[16];
        int dst[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) {
            const int d = d0 + (e >> 1), h = e & 1;
            const int r = lane + 32 * h, k = (r + d) & 63;
            dst[e] = -1;
            v[e] = 0.0;
            if (r < n && k < n && (d < 32 || h == 0)) {
                v[e] = pair_cov64(J, P, own[h], nb[k]);
                const int lo = r < k ? r : k, hi = r < k ? k : r;
                if (CORR) v[e] = __dmul_rn(v[e], __dmul_rn(sg[hi], sg[lo]));
                dst[e] = cs[hi] + lo;
            }
        }
#pragma unroll
        for (int e = 0; e < 16; ++e)
            if (dst[e] >= 0) U[dst[e]] = v[e];
    }
    __syncwarp();
}

// Factorises and solves one system (weights of rows lane, lane + 32 in w0,
// w1); returns the status.  CORR scales entry (i, k) by sg[k] sg[i]
// (corellogramed_weights_3, my_kriging_weights.h:308-317; b is scaled by
// the caller).
template <bool CORR>
__device__ int exact64_core(const DevJob &J, const DevPlan &P, Exact64Smem &S, const int *cs,
                            int lane, const Node64 &d, const double *sg, double &w0_out, double &w1_out) {
    const int n = d.n;
    const bool ordinary = J.kind == 0;
    double *U = S.U;
    build_packed<CORR>(J, P, U, S.nb, cs, n, lane, sg);
    const int k0 = lane, k1 = lane + 32;  // the lane's columns in the factorisation
    const double a_diag = __ldg(P.table);  // A(k,k) = C(0)
    // diagonal slots and pads of the lane's columns are zero until their step
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int k = lane + 32 * h;
        U[cs[k] + k] = 0.0;
        if (!(k & 1)) U[cs[k] + k + 1] = 0.0;
    }
    __syncwarp();
    const double *c0 = U + cs[k0];
    const double *c1 = U + cs[k1];
    int info = 0;
    double dg0 = 0.0, rc0 = 0.0, dg1 = 0.0, rc1 = 0.0;  // U(k,k) and RN(1/U(k,k)) of the lane's columns
    double xa0 = d.b[0], xa1 = d.b[1], xb0 = 1.0, xb1 = 1.0;
    // DPOTF2 'U' step j, left-looking like the reference: the sums
    // t = sum_{i<j} U(i,k) U(i,j) (DDOT for k = j, DGEMV for k > j) run over i in
    // ascending order from +0, each lane over its own columns while column j
    // is broadcast; an odd j pairs row j, whose slot in column j is still
    // zero.  Every lane runs every instruction of a step: the pivot's square
    // root and reciprocal and the forward division are computed by all lanes
    // from broadcast values (the same operations the owner would do), which
    // keeps the warp converged.
    for (int j = 0; j < n; ++j) {
        const bool lo = j < 32;  // the lane's first column is still open
        const int owner = j & 31;
        const bool mine = lane == owner;
        const double2 *uj = reinterpret_cast<const double2 *>(U + cs[j]);
        const double2 *a0p = reinterpret_cast<const double2 *>(c0);
        const double2 *a1p = reinterpret_cast<const double2 *>(c1);
        double t0 = 0.0, t1 = 0.0;
        const int pairs = (j + 1) >> 1;
        if (lo) {
            for (int q = 0; q < pairs; ++q) {
                const double2 u = uj[q], a0 = a0p[q], a1 = a1p[q];
                t0 = __dadd_rn(t0, __dmul_rn(a0.x, u.x));
                t1 = __dadd_rn(t1, __dmul_rn(a1.x, u.x));
                t0 = __dadd_rn(t0, __dmul_rn(a0.y, u.y));
                t1 = __dadd_rn(t1, __dmul_rn(a1.y, u.y));
            }
        } else {
            for (int q = 0; q < pairs; ++q) {
                const double2 u = uj[q], a1 = a1p[q];
                t1 = __dadd_rn(t1, __dmul_rn(a1.x, u.x));
                t1 = __dadd_rn(t1, __dmul_rn(a1.y, u.y));
            }
        }
        // every lane has read column j's diagonal slot before it is written
        __syncwarp();
        const double tj = __shfl_sync(FULL_MASK, lo ? t0 : t1, owner);
        const double ajj = __dsub_rn(CORR ? __dmul_rn(a_diag, __dmul_rn(sg[j], sg[j])) : a_diag, tj);
        if (!(ajj > 0.0)) {
            info = j + 1;
            break;
        }
        const double ujj = dsqrt64(ajj);
        const double rinv = drcp64(ujj);
        if (mine) {
            U[cs[j] + j] = ujj;
            if (lo) {
                dg0 = ujj;
                rc0 = rinv;
            } else {
                dg1 = ujj;
                rc1 = rinv;
            }
        }
        // forward substitution U^T y = b, row j final: y_j = x_j / u_jj
        const double xaj = __shfl_sync(FULL_MASK, lo ? xa0 : xa1, owner);
        const double ya = div_by_rcp(xaj, ujj, rinv);
        double yb = 0.0;
        if (ordinary) yb = div_by_rcp(__shfl_sync(FULL_MASK, lo ? xb0 : xb1, owner), ujj, rinv);
        if (mine) {
            if (lo) {
                xa0 = ya;
                xb0 = yb;
            } else {
                xa1 = ya;
                xb1 = yb;
            }
        }
        // row j of U: u_jk = (a_jk - t) / u_jj for the lane's columns k > j,
        // then x_k -= u_jk y_j
        if (lo && k0 > j) {
            double v = U[cs[k0] + j];
            if (j > 0) v = __dadd_rn(v, -t0);
            const double v0 = __dmul_rn(rinv, v);
            U[cs[k0] + j] = v0;
            xa0 = __dsub_rn(xa0, __dmul_rn(v0, ya));
            if (ordinary) xb0 = __dsub_rn(xb0, __dmul_rn(v0, yb));
        }
        if (k1 > j) {
            double v = U[cs[k1] + j];
            if (j > 0) v = __dadd_rn(v, -t1);
            const double v1 = __dmul_rn(rinv, v);
            U[cs[k1] + j] = v1;
            xa1 = __dsub_rn(xa1, __dmul_rn(v1, ya));
            if (ordinary) xb1 = __dsub_rn(xb1, __dmul_rn(v1, yb));
        }
        __syncwarp();
    }
    double w0 = 0.0, w1 = 0.0;
    int status = ST_SUCCESS;
    const int n0 = n < 32 ? n : 32;  // rows held in the lanes' first halves
    if (info != 0) {
        status = ST_SINGULAR;
    } else {
        // DPOTRS back substitution U x = y (DTRSM column form, k descending):
        // x_k /= u_kk where x_k != 0, then x_i -= x_k u_ik for i < k.
        for (int k = n - 1; k >= 0; --k) {
            const int owner = k & 31;
            const bool hi = k >= 32;
            const double ukk = __shfl_sync(FULL_MASK, hi ? dg1 : dg0, owner);
            const double rk = __shfl_sync(FULL_MASK, hi ? rc1 : rc0, owner);
            double va = __shfl_sync(FULL_MASK, hi ? xa1 : xa0, owner);
            double vb = ordinary ? __shfl_sync(FULL_MASK, hi ? xb1 : xb0, owner) : 0.0;
            const bool nza = va != 0.0, nzb = vb != 0.0;
            if (nza) va = div_by_rcp(va, ukk, rk);
            if (nzb) vb = div_by_rcp(vb, ukk, rk);
            if (lane == owner) {
                if (hi) {
                    xa1 = va;
                    xb1 = vb;
                } else {
                    xa0 = va;
                    xb0 = vb;
                }
            }
            const double *uk = U + cs[k];
            if (k0 < k) {
                const double u = uk[k0];
                if (nza) xa0 = __dsub_rn(xa0, __dmul_rn(va, u));
                if (nzb) xb0 = __dsub_rn(xb0, __dmul_rn(vb, u));
            }
            if (k1 < k) {
                const double u = uk[k1];
                if (nza) xa1 = __dsub_rn(xa1, __dmul_rn(va, u));
                if (nzb) xb1 = __dsub_rn(xb1, __dmul_rn(vb, u));
            }
        }
        if (ordinary) {
            // SumSK, SumOnes in row order (my_kriging_weights.h), then
            // mu = (SumSK - 1) / SumOnes and w = x_sk - mu x_ones
            double ssk = 0.0, son = 0.0;
            for (int i = 0; i < n0; ++i) {
                ssk = __dadd_rn(ssk, __shfl_sync(FULL_MASK, xa0, i));
                son = __dadd_rn(son, __shfl_sync(FULL_MASK, xb0, i));
            }
            for (int i = 32; i < n; ++i) {
                ssk = __dadd_rn(ssk, __shfl_sync(FULL_MASK, xa1, i - 32));
                son = __dadd_rn(son, __shfl_sync(FULL_MASK, xb1, i - 32));
            }
            const double mu = __ddiv_rn(__dsub_rn(ssk, 1.0), son);
            w0 = __dsub_rn(xa0, __dmul_rn(mu, xb0));
            w1 = __dsub_rn(xa1, __dmul_rn(mu, xb1));
        } else {
            w0 = xa0;
            w1 = xa1;
        }
    }
    w0_out = w0;
    w1_out = w1;
    return status;
}

__device__ void exact64_system(const DevJob &J, const DevPlan &P, Exact64Smem &S, const int *cs, int node,
                               int lane, const Node64 &d) {
    const int n = d.n;
    const bool ordinary = J.kind == 0;
    const int n0 = n < 32 ? n : 32;
    double w0, w1;
    const int status = exact64_core<false>(J, P, S, cs, lane, d, nullptr, w0, w1);
    double variance = -1.0;
    if (J.variance && status == ST_SUCCESS) {
        double v = P.c0;
        const double p0 = __dmul_rn(w0, d.b[0]), p1 = __dmul_rn(w1, d.b[1]);
        for (int i = 0; i < n0; ++i) v = __dsub_rn(v, __shfl_sync(FULL_MASK, p0, i));
        for (int i = 32; i < n; ++i) v = __dsub_rn(v, __shfl_sync(FULL_MASK, p1, i - 32));
        if (ordinary) v = __dsub_rn(v, row_val(w0, w1, n - 1));
        variance = v;
    }
    write_outputs64(J, P, node, lane, d, status, w0, w1, variance);
}

// One node of the exact path; returns whether a system was solved.
__device__ __forceinline__ bool exact64_node(const DevJob &J, const DevPlan &P, Exact64Smem &S, const int *cs,
                                             const NodeFetch &cur, int lane) {
    if (copy_informed64(J, cur, lane)) return false;
    const Node64 d = load_node64(J, P, S.nb, cur, lane);
    if (d.n <= 0) {
        write_outputs64(J, P, cur.node, lane, d, ST_NO_NEIGHBOURS, 0.0, 0.0, -1.0);
        return false;
    }
    exact64_system(J, P, S, cs, cur.node, lane, d);
    return true;
}

// One speculative round of sequential simulation (33-64 neighbours): one
// warp per pending node of window buffer `cur`.
__global__ void __launch_bounds__(WARPS64_BLOCK * 32) k_sgs_try64(DevJob J, DevPlan P, SgsState G, int cur) {
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    __shared__ int s_cs[N64];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int k = threadIdx.x; k < N64; k += blockDim.x) s_cs[k] = col_start_c(k);
    __syncthreads();
    Exact64Smem &S = reinterpret_cast<Exact64Smem *>(dyn_smem)[warp];
    const int ntry = G.ctl->ntry;
    const int *win = cur ? G.win1 : G.win0;
    // the round's tries are handed out one at a time as warps free up
    int slot, rank;
    while (sgs_next_try(G, win, ntry, lane, slot, rank)) {
        const int node = G.nodes[rank];
        int cnt;
        const int blocker = template_node_spec(J, P, G, node, rank, lane, J.nb + (long long)node * P.nmax, cnt);
        if (lane == 0 && blocker < 0) J.nbcount[node] = cnt;
        __syncwarp();
        if (blocker < 0) {
            const NodeFetch f = fetch_node(J, P, node, lane);
            exact64_node(J, P, S, s_cs, f, lane);
            __syncwarp();
            if (lane == 0) sgs_value(J, node, G.xp[rank]);
        }
        if (lane == 0) {
            G.ok[slot] = blocker < 0;
            if (blocker >= 0) G.blocker[rank] = blocker;
        }
        __syncwarp();
    }
}

// Every node, for the jobs the tiled kernels do not take (tile_takes).
__global__ void __launch_bounds__(WARPS64_BLOCK * 32) k_solve_exact64(DevJob J, DevPlan P) {
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    __shared__ int s_cs[N64];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int k = threadIdx.x; k < N64; k += blockDim.x) s_cs[k] = col_start_c(k);
    __syncthreads();
    Exact64Smem &S = reinterpret_cast<Exact64Smem *>(dyn_smem)[warp];
    unsigned long long solved = 0;
    // warps take up to CHUNK64 consecutive nodes at a time from a per-job
    // counter (the next chunk taken while the current one's last node is
    // solved), so none waits on a fixed share at the end
    const int csize = chunk_nodes(J, CHUNK64, WARPS64_BLOCK);
    int chunk = take_chunk64(J, lane, csize);
    long long it = chunk_first(chunk, J.size);
    NodeFetch cur = fetch_node(J, P, it < J.size ? (int)it : -1, lane);
    while (it < J.size) {
        long long nx = it + 1;
        int nchunk = chunk;
        if (nx == (long long)chunk + csize) {
            nchunk = take_chunk64(J, lane, csize);
            nx = chunk_first(nchunk, J.size);
        }
        const NodeFetch next = fetch_node(J, P, nx < J.size ? (int)nx : -1, lane);
        solved += exact64_node(J, P, S, s_cs, cur, lane);
        __syncwarp();
        cur = next;
        it = nx;
        chunk = nchunk;
    }
    if (lane == 0 && solved) atomicAdd(J.n_fp64, solved);
}

// Fused search + solve (one warp per block): template search of a 32-node
// segment, then the segment's systems, as in the 32-neighbour fused kernel.
__global__ void __launch_bounds__(32) k_fused64(DevJob J, DevPlan P) {
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    __shared__ int s_cs[N64];
    __shared__ int delta_sm[32];
    const int lane = threadIdx.x & 31;
    for (int k = threadIdx.x; k < N64; k += blockDim.x) s_cs[k] = col_start_c(k);
    __syncthreads();
    const long long total = (long long)P.nseg * J.ny * J.nz;
    unsigned long long solved = 0;
    for (long long segi = blockIdx.x; segi < total; segi += gridDim.x) {
        const int base = template_segment(J, P, segi, lane, delta_sm);
        __syncwarp();
        const int x0 = (int)(segi % P.nseg) * 32;
        const int cnt = min(32, J.nx - x0);
        NodeFetch next = fetch_node(J, P, base, lane);
        for (int b = 0; b < cnt; ++b) {
            const NodeFetch cur = next;
            next = fetch_node(J, P, b + 1 < cnt ? base + b + 1 : -1, lane);
            solved += exact64_node(J, P, *reinterpret_cast<Exact64Smem *>(dyn_smem), s_cs, cur, lane);
            __syncwarp();
        }
    }
    if (lane == 0 && solved) atomicAdd(J.n_fp64, solved);
}

constexpr size_t SMEM64_EXACT = sizeof(Exact64Smem) * WARPS64_BLOCK;

// ---------------------------------------------------------------------------
// Sequential indicator simulation with categories of up to 64 neighbours
// (the 32-neighbour kernel's rules, k_sis_try32 in solve32.cu).

struct Sis64Smem {
    Exact64Smem e;
    double sg[N64];  // the rows' sigma (correlogram weights)
};

__device__ __forceinline__ Node64 sis_load64(const DevJob &J, const DevPlan &P, Sis64Smem &S, int node,
                                             const int *list, int n, int k, double sgc, int lane) {
    Node64 d;
    d.n = n;
    int x0, y0, z0;
    node_xyz(J, node, x0, y0, z0);
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int row = lane + 32 * r;
        d.dv[r] = 0.f;
        d.code[r] = -1;
        d.b[r] = 0.0;
        double sg = 0.0;
        int4 o = make_int4(0, 0, 0, 0);
        if (row < n) {
            const int cell = list[row];
            int qx, qy, qz;
            node_xyz(J, cell, qx, qy, qz);
            o.x = qx - x0;
            o.y = qy - y0;
            o.z = qz - z0;
            o.w = o.z * P.syx + o.y * P.sx + o.x;
            const float m = sis_mean(J, k, cell);
            d.dv[r] = __fsub_rn(J.codes[cell] == k ? 1.f : 0.f, m);
            d.b[r] = cov_lin(P, o.x, o.y, o.z, o.w, J.err);
            if (J.sis_corr) {
                sg = sis_sigma(m);
                d.b[r] = __dmul_rn(d.b[r], __dmul_rn(sg, sgc));
            }
        }
        S.e.nb[row] = o;
        S.sg[row] = sg;
    }
    __syncwarp();
    return d;
}

__global__ void __launch_bounds__(WARPS64_BLOCK * 32) k_sis_try64(DevJob J, const DevPlan *plans, SgsState G, int cur) {
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    __shared__ int s_cs[N64];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int k = threadIdx.x; k < N64; k += blockDim.x) s_cs[k] = col_start_c(k);
    __syncthreads();
    Sis64Smem &S = reinterpret_cast<Sis64Smem *>(dyn_smem)[warp];
    const int ntry = G.ctl->ntry;
    const int *win = cur ? G.win1 : G.win0;
    const int cats = J.K == 2 ? 1 : J.K;
    // the round's tries are handed out one at a time as warps free up
    int slot, rank;
    while (sgs_next_try(G, win, ntry, lane, slot, rank)) {
        const int node = G.nodes[rank];
        int *list = J.nb + (long long)node * J.nb_stride;
        float *probs = J.probs + (long long)node * J.K;
        int blocker = -1;
        for (int k = 0; k < cats; ++k) {
            const DevPlan &P = plans[k];
            int cnt;
            blocker = template_node_spec(J, P, G, node, rank, lane, list, cnt);
            if (blocker >= 0) break;
            __syncwarp();
            const float mc = sis_mean(J, k, node);
            double prob = (double)mc;
            if (cnt > 0) {
                const double sgc = J.sis_corr ? sis_sigma(mc) : 0.0;
                const Node64 d = sis_load64(J, P, S, node, list, cnt, k, sgc, lane);
                double w0, w1;
                const int status =
                    J.sis_corr ? exact64_core<true>(J, P, S.e, s_cs, lane, d, S.sg, w0, w1)
                               : exact64_core<false>(J, P, S.e, s_cs, lane, d, nullptr, w0, w1);
                if (status == ST_SUCCESS) {
                    const double t0 = __dmul_rn(w0, (double)d.dv[0]), t1 = __dmul_rn(w1, (double)d.dv[1]);
                    prob = rows_dsum((double)mc, t0, t1, cnt);
                }
            }
            if (lane == 0) {
                probs[k] = __double2float_rn(prob);
                if (J.K == 2) probs[1] = __double2float_rn(__dsub_rn(1.0, prob));
            }
            __syncwarp();
        }
        if (lane == 0) sis_finish(J, G, node, rank, slot, blocker);
        __syncwarp();
    }
}

}  // namespace

// The tile of a job's systems by its largest neighbour count.  Up to 56: 16
// lanes a system, 2 systems a warp (8 lanes, 4 systems: S36 31.1, 40 35.9, 48
// 84 ms, the factors of too few systems fit an SM's shared memory), one-warp
// blocks, as many as the factors leave room for (12 up to 40 neighbours, then
// 8 and 7).  Above, two factors a warp leave room for 5 warps; 32 lanes a
// system, 8 x 4, take half the shared memory and hold 8 warps, whose 3 200
// more instructions a system (the pivot chain is shared by fewer) cost less
// than the better occupancy gives: issue slots in use 48 % for 31 %.  At 56
// and below they cost more (56: 85.2, 48: 61.0, 40: 43.8 ms).  Solve of SK
// 256x256x64 (4.15 M systems) with the neighbour count set, in ms (one system
// a warp, two columns a lane): 36: 28.8   40: 34.0 [149.6]   44: 39.1   48:
// 45.1 [181.7]   52: 66.2   56: 76.3 [211.3]   64: 106.1 [241.7], 123.2 with
// 16 lanes; LVM 512x512x32 (7.5 M systems, 64) 175.7 [327], with 16
// lanes 244.  Panels (row blocks whose sums are kept open together) two blocks
// narrower / wider on the same job: 36: 28.4 / 29.4   40: 33.1 / 34.6   44: 40.6
// / 41.3   48: 45.6 / 48.7   52: 70.5 / 71.3   56: 78.5 / 78.8   64: 111.7 / 109.5;
// at 36 and 40, where the panel of 4 spills 120 and 196 bytes, the narrower one
// would be 2 % faster.
void launch_solve64(const DevJob &J, const DevPlan &P, cudaStream_t s, int blocks_per_sm) {
    const int b = blocks_per_sm;
    if (!tile_takes(P)) {
        const long long g = persistent_grid((const void *)k_solve_exact64, WARPS64_BLOCK * 32, SMEM64_EXACT, b,
                                            (J.size + WARPS64_BLOCK - 1) / WARPS64_BLOCK);
        k_solve_exact64<<<(unsigned)g, WARPS64_BLOCK * 32, SMEM64_EXACT, s>>>(J, P);
    } else if (P.nmax <= 36) {
        launch_tile<TileGeom<36, 4, 4, 4>, 1, 12>(J, P, s, b);
    } else if (P.nmax <= 40) {
        launch_tile<TileGeom<40, 4, 4, 4>, 1, 12>(J, P, s, b);
    } else if (P.nmax <= 44) {
        launch_tile<TileGeom<44, 4, 4, 6>, 1, 8>(J, P, s, b);
    } else if (P.nmax <= 48) {
        launch_tile<TileGeom<48, 4, 4, 6>, 1, 8>(J, P, s, b);
    } else if (P.nmax <= 52) {
        launch_tile<TileGeom<52, 4, 4, 4>, 1, 7>(J, P, s, b);
    } else if (P.nmax <= 56) {
        launch_tile<TileGeom<56, 4, 4, 4>, 1, 7>(J, P, s, b);
    } else {
        launch_tile<TileGeom<64, 8, 4, 4>, 2, 4>(J, P, s, b);
    }
}

void launch_sgs_try64(const DevJob &J, const DevPlan &P, const SgsState &G, int cur, cudaStream_t s) {
    const long long g = persistent_grid((const void *)k_sgs_try64, WARPS64_BLOCK * 32, SMEM64_EXACT, 0, 1LL << 30);
    k_sgs_try64<<<(unsigned)g, WARPS64_BLOCK * 32, SMEM64_EXACT, s>>>(J, P, G, cur);
}

void launch_sis_try64(const DevJob &J, const DevPlan *plans, const SgsState &G, int cur, cudaStream_t s) {
    const size_t smem = sizeof(Sis64Smem) * WARPS64_BLOCK;
    const long long g = persistent_grid((const void *)k_sis_try64, WARPS64_BLOCK * 32, smem, 0, 1LL << 30);
    k_sis_try64<<<(unsigned)g, WARPS64_BLOCK * 32, smem, s>>>(J, plans, G, cur);
}

void launch_fused64(const DevJob &J, const DevPlan &P, cudaStream_t s, int blocks_per_sm) {
    const long long segs = (long long)P.nseg * J.ny * J.nz;
    if (segs <= 0) return;
    const long long g = persistent_grid((const void *)k_fused64, 32, sizeof(Exact64Smem), blocks_per_sm, segs);
    k_fused64<<<(unsigned)g, 32, sizeof(Exact64Smem), s>>>(J, P);
}

}  // namespace hpgl_b200
