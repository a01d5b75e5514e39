// Per-node solves for systems of at most 32 neighbours, FP64 in the
// reference's exact operation order (my_kriging_weights.h:26-255 over LAPACK
// DPOTF2 / DPOTRS).
//
//   k_solve_tile     (tile_solve.cuh) several systems a warp, persistent over
//                    the grid's nodes: every kriging job's solve.
//   exact_core       one system a warp, lane k holding column k in registers,
//                    the finished part of column j broadcast through shared
//                    memory as 16-byte pairs for the dot products of step j:
//                    sequential simulation (a node's search and system in one
//                    warp, one node at a time), the fused search + solve
//                    kernel, and the jobs the tiled kernels do not take
//                    (k_solve_exact32).
#include "device_common.cuh"
#include "search_common.cuh"
#include "tile_solve.cuh"

namespace hpgl_b200 {

namespace {

constexpr int N32 = 32;
constexpr int WARPS32 = 4;

// Per-warp shared memory; NA doubles of system storage (columns of 34: NC *
// 34 for systems of at most NC neighbours).
template <int NA>
struct SysSmemN {
    double A[NA];           // in-place factor (column k at k*34)
    double vd[N32];         // double vector broadcast
    float vf[2][N32];       // float vector broadcast
    float row[2][N32];      // simulation: the neighbour list
    int4 nb[N32];           // neighbour offsets from the node (x, y, z, table offset)
};
using SysSmem = SysSmemN<N32 * 34>;
// systems of at most 16 neighbours (sequential simulation): half the
// registers and shared memory, twice the warps per SM
constexpr int N16 = 16;
using SysSmem16 = SysSmemN<N16 * 34>;

// Per-node prologue.  Returns n (neighbour count) and
// fills the lane's neighbour data; the system itself is built separately.
struct NodeData {
    int n;
    float dv;   // cont: value - mean of row `lane` (float, combiner.h:18-22)
    int code;   // IK: category code of row `lane`
    double b;   // b_lane = C(x_lane - x0)
    int ox, oy, oz, lin;  // offset of neighbour `lane` from the node, and its table offset
};

template <typename SM>
__device__ __forceinline__ NodeData load_node(const DevJob &J, const DevPlan &P, SM &S, const NodeFetch &f,
                                              int lane) {
    NodeData d;
    const int node = f.node;
    d.n = f.n;
    int x0, y0, z0;
    node_xyz(J, node, x0, y0, z0);
    d.dv = 0.f;
    d.code = -1;
    d.b = 0.0;
    int ox = 0, oy = 0, oz = 0;
    if (lane < d.n) {
        const int cell = f.cell;
        int qx, qy, qz;
        node_xyz(J, cell, qx, qy, qz);
        ox = qx - x0;
        oy = qy - y0;
        oz = qz - z0;
        if (is_cont(J.kind)) {
            const float m = J.kind == 1 ? J.sk_mean_f : (J.kind == 2 ? J.mean[cell] : 0.f);
            d.dv = __fsub_rn(J.values[cell], m);
        } else {
            d.code = J.codes[cell];
        }
        d.b = cov_at(P, ox, oy, oz, J.err);
    }
    d.ox = ox;
    d.oy = oy;
    d.oz = oz;
    d.lin = oz * P.syx + oy * P.sx + ox;
    S.nb[lane] = make_int4(ox, oy, oz, d.lin);
    __syncwarp();
    return d;
}

// init + t_0 + t_1 + ... + t_{n-1} in that order, t_i = `term` of lane i,
// computed by lane 0 from 16-byte reads of a shared buffer (valid on lane 0).
__device__ __forceinline__ float seq_fsum(float init, float term, int n, float *buf, int lane) {
    buf[lane] = term;
    __syncwarp();
    float r = init;
    if (lane == 0) {
        const float4 *b4 = reinterpret_cast<const float4 *>(buf);
#pragma unroll
        for (int q = 0; q < N32 / 4; ++q) {
            if (4 * q < n) {
                const float4 v = b4[q];
                r = __fadd_rn(r, v.x);
                if (4 * q + 1 < n) r = __fadd_rn(r, v.y);
                if (4 * q + 2 < n) r = __fadd_rn(r, v.z);
                if (4 * q + 3 < n) r = __fadd_rn(r, v.w);
            }
        }
    }
    __syncwarp();
    return r;
}
__device__ __forceinline__ double seq_dsum(double init, double term, int n, double *buf, int lane) {
    buf[lane] = term;
    __syncwarp();
    double r = init;
    if (lane == 0) {
        const double2 *b2 = reinterpret_cast<const double2 *>(buf);
#pragma unroll
        for (int q = 0; q < N32 / 2; ++q) {
            if (2 * q < n) {
                const double2 v = b2[q];
                r = __dadd_rn(r, v.x);
                if (2 * q + 1 < n) r = __dadd_rn(r, v.y);
            }
        }
    }
    __syncwarp();
    return r;
}

// Outputs of one solved (or failed) system: weights w (row `lane`), status.
// The estimate sums run on lane 0 in neighbour order (combiner.h:9-24:
// float terms summed in float; median IK in double), which is also the only
// lane that stores them.
template <typename SM>
__device__ __forceinline__ void write_outputs(const DevJob &J, const DevPlan &P, SM &S, int node, int lane,
                                              const NodeData &d, int status, double w, double variance) {
    const long long slot = (long long)node * J.status_stride + J.status_offset;
    const bool success = status == ST_SUCCESS;
    const int n = d.n;
    if (J.weights && n > 0 && lane < n) J.weights[slot * P.nmax + lane] = w;
    if (J.variance && lane == 0) J.variance[slot] = success ? variance : -1.0;
    if (lane == 0) J.status[slot] = (int8_t)status;
    if (is_cont(J.kind)) {
        if (success) {
            const float term = __double2float_rn(__dmul_rn(w, (double)d.dv));
            const float m0 = J.kind == 1 ? J.sk_mean_f : (J.kind == 2 ? J.mean[node] : 0.f);
            const float res = seq_fsum(m0, term, n, S.vf[0], lane);
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
                const float term = __double2float_rn(__dmul_rn(w, (double)__fsub_rn(d.code == k ? 1.f : 0.f, pk)));
                prob = seq_fsum(pk, term, n, S.vf[0], lane);
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
            const double term = __dmul_rn(w, (double)__fsub_rn(d.code == 1 ? 1.f : 0.f, m));
            prob = seq_dsum(prob, term, n, S.vd, lane);
        }
        if (lane == 0) {
            J.probs[node] = (float)prob;
            J.out_codes[node] = ((float)prob <= 0.5f) ? 0 : 1;
            J.out_mask[node] = 1;
        }
    }
}

__device__ __forceinline__ bool copy_informed(const DevJob &J, const NodeFetch &f, int lane) {
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

// ---------------------------------------------------------------------------

// IEEE square root and reciprocal (one lane per factorisation step).
__device__ __noinline__ double dsqrt_rn(double a) { return __dsqrt_rn(a); }
__device__ __noinline__ double drcp_rn(double a) { return __drcp_rn(a); }

// Factorises and solves one system (weights of row `lane` in w); returns the
// status.  Lane k gathers column k of the upper triangle straight into
// registers.  CORR scales entry (i, k) by sg_k sg_i, sg the lanes' sigma
// (corellogramed_weights_3, my_kriging_weights.h:308-317; b is scaled by the
// caller).
template <bool CORR, int NC = N32, typename SM>
__device__ __forceinline__ int exact_core(const DevJob &J, const DevPlan &P, SM &S, int lane, const NodeData &d,
                                          double sg, double &w_out) {
    constexpr int LD = 34;
    const int n = d.n;
    const bool ordinary = J.kind == 0;
    double c[NC];
#pragma unroll
    for (int i = 0; i < NC; ++i) {
        // A(i, lane) = C(x_i - x_lane) for i <= lane (my_kriging_weights.h:53);
        // neighbour i's offsets are one broadcast read of S.nb
        const int4 q = S.nb[i];
        const double si = CORR ? __shfl_sync(FULL_MASK, sg, i) : 0.0;
        c[i] = 0.0;
        if (i <= lane && lane < n) {
            c[i] = cov_lin(P, q.x - d.ox, q.y - d.oy, q.z - d.oz, q.w - d.lin, J.err);
            if (CORR) c[i] = __dmul_rn(c[i], __dmul_rn(sg, si));
        }
    }
    // DPOTF2 'U': column j, ajj = a_jj - sum_{i<j} a_ij^2; a_jk += -sum a_ij a_ik;
    // a_jk *= 1/ajj.  Finished entries U(j,k) go to S.A (column k at k*34)
    // for the broadcasts and for the transposed reads of the back substitution.
    int info = 0;
    double my_rcp = 0.0;  // RN(1/U(lane,lane))
#pragma unroll
    for (int j = 0; j < NC; ++j) {
        if (j >= n) break;
        double t = 0.0;
        const double2 *cj = reinterpret_cast<const double2 *>(S.A + j * LD);
#pragma unroll
        for (int q = 0; q < (j + 1) / 2; ++q) {
            const double2 u = cj[q];
            t = __dadd_rn(t, __dmul_rn(c[2 * q], u.x));
            if (2 * q + 1 < j) t = __dadd_rn(t, __dmul_rn(c[2 * q + 1], u.y));
        }
        int fail = 0;
        double rinv = 0.0;
        if (lane == j) {
            double ajj = __dsub_rn(c[j], t);
            if (!(ajj > 0.0)) {
                fail = 1;
            } else {
                ajj = dsqrt_rn(ajj);
                rinv = drcp_rn(ajj);
            }
            c[j] = ajj;
            S.A[j * LD + j] = ajj;
            my_rcp = rinv;
        }
        fail = __shfl_sync(FULL_MASK, fail, j);
        if (fail) {
            info = j + 1;
            break;
        }
        rinv = __shfl_sync(FULL_MASK, rinv, j);
        if (lane > j && lane < NC) {  // the lane's column exists (NC * 34 doubles of S.A)
            double v = c[j];
            if (j > 0) v = __dadd_rn(v, -t);
            v = __dmul_rn(rinv, v);
            c[j] = v;
            S.A[lane * LD + j] = v;
        }
        __syncwarp();
    }
    double w = 0.0;
    int status = ST_SUCCESS;
    if (info != 0) {
        status = ST_SINGULAR;
    } else {
        // DPOTRS 'U': U^T y = b (dot form, k ascending), then U x = y (column form).
        double xa = d.b, xb = 1.0;
#pragma unroll
        for (int i = 0; i < NC; ++i) {
            if (i >= n) break;
            double ya = 0.0, yb = 0.0;
            if (lane == i) {
                ya = div_by_rcp(xa, c[i], my_rcp);
                xa = ya;
                if (ordinary) {
                    yb = div_by_rcp(xb, c[i], my_rcp);
                    xb = yb;
                }
            }
            ya = __shfl_sync(FULL_MASK, ya, i);
            if (ordinary) yb = __shfl_sync(FULL_MASK, yb, i);
            if (lane > i) {
                xa = __dsub_rn(xa, __dmul_rn(c[i], ya));
                if (ordinary) xb = __dsub_rn(xb, __dmul_rn(c[i], yb));
            }
        }
        __syncwarp();
        for (int k = n - 1; k >= 0; --k) {
            double va = __shfl_sync(FULL_MASK, xa, k);
            double vb = ordinary ? __shfl_sync(FULL_MASK, xb, k) : 0.0;
            const bool nza = va != 0.0, nzb = vb != 0.0;
            if (lane == k) {
                const double ukk = S.A[k * LD + k];
                if (nza) xa = div_by_rcp(xa, ukk, my_rcp);
                if (ordinary && nzb) xb = div_by_rcp(xb, ukk, my_rcp);
            }
            va = __shfl_sync(FULL_MASK, xa, k);
            if (ordinary) vb = __shfl_sync(FULL_MASK, xb, k);
            if (lane < k) {
                const double u = S.A[k * LD + lane];
                if (nza) xa = __dsub_rn(xa, __dmul_rn(va, u));
                if (ordinary && nzb) xb = __dsub_rn(xb, __dmul_rn(vb, u));
            }
        }
        if (ordinary) {
            const double ssk = __shfl_sync(FULL_MASK, seq_dsum(0.0, lane < n ? xa : 0.0, n, S.vd, lane), 0);
            const double son = __shfl_sync(FULL_MASK, seq_dsum(0.0, lane < n ? xb : 0.0, n, S.vd, lane), 0);
            const double mu = __ddiv_rn(__dsub_rn(ssk, 1.0), son);
            w = __dsub_rn(xa, __dmul_rn(mu, xb));
        } else {
            w = xa;
        }
    }
    w_out = w;
    return status;
}

// Solves and writes the outputs of one system.
template <int NC = N32, typename SM>
__device__ __forceinline__ void exact_system(const DevJob &J, const DevPlan &P, SM &S, int node, int lane,
                                             const NodeData &d) {
    const int n = d.n;
    const bool ordinary = J.kind == 0;
    double w;
    const int status = exact_core<false, NC>(J, P, S, lane, d, 0.0, w);
    double variance = -1.0;
    if (J.variance && status == ST_SUCCESS) {
        // c0 - p_0 - p_1 - ... (my_kriging_weights.h): subtracting p is adding -p
        double v = seq_dsum(P.c0, -__dmul_rn(w, d.b), n, S.vd, lane);
        if (ordinary) v = __dsub_rn(v, __shfl_sync(FULL_MASK, w, n - 1));
        variance = v;
    }
    write_outputs(J, P, S, node, lane, d, status, w, variance);
}

// One node of the exact path; returns whether a system was solved.
template <int NC = N32, typename SM>
__device__ __forceinline__ bool exact32_node(const DevJob &J, const DevPlan &P, SM &S, const NodeFetch &cur,
                                             int lane) {
    if (copy_informed(J, cur, lane)) return false;
    const NodeData d = load_node(J, P, S, cur, lane);
    if (d.n <= 0) {
        write_outputs(J, P, S, cur.node, lane, d, ST_NO_NEIGHBOURS, 0.0, -1.0);
        return false;
    }
    exact_system<NC>(J, P, S, cur.node, lane, d);
    return true;
}

// Every node, for the jobs the tiled kernels do not take (tile_takes).
// Warps take up to 32 consecutive nodes at a time from the per-job counter.
__global__ void __launch_bounds__(WARPS32 * 32) k_solve_exact32(DevJob J, DevPlan P) {
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    SysSmem &S = reinterpret_cast<SysSmem *>(dyn_smem)[warp];
    unsigned long long solved = 0;
    const int csize = chunk_nodes(J, 32, WARPS32);
    int chunk = 0;
    if (lane == 0) chunk = atomicAdd(J.node_next, csize);
    chunk = __shfl_sync(FULL_MASK, chunk, 0);
    long long it = chunk_first(chunk, J.size);
    NodeFetch cur = fetch_node(J, P, it < J.size ? (int)it : -1, lane);
    while (it < J.size) {
        long long nx = it + 1;
        int nchunk = chunk;
        if (nx == (long long)chunk + csize) {
            int c = 0;
            if (lane == 0) c = atomicAdd(J.node_next, csize);
            nchunk = __shfl_sync(FULL_MASK, c, 0);
            nx = chunk_first(nchunk, J.size);
        }
        const NodeFetch next = fetch_node(J, P, nx < J.size ? (int)nx : -1, lane);
        solved += exact32_node(J, P, S, cur, lane);
        __syncwarp();
        cur = next;
        it = nx;
        chunk = nchunk;
    }
    if (lane == 0 && solved) atomicAdd(J.n_fp64, solved);
}

// Fused search + solve: each warp takes 32-node x-segments, runs the template
// search for the segment's template-path nodes (lists to J.nb, still in L2),
// then solves the segment's nodes one after the other -- the clusterizer-path
// nodes' lists come from the clusterizer search launched before.  Warps in
// the search phase (memory latency) and in the solve phase (FP pipes)
// overlap on every SM.
__global__ void __launch_bounds__(WARPS32 * 32) k_fused32(DevJob J, DevPlan P) {
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    __shared__ int delta_sm[WARPS32][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    SysSmem &S = reinterpret_cast<SysSmem *>(dyn_smem)[warp];
    const long long total = (long long)P.nseg * J.ny * J.nz;
    const long long stride = (long long)gridDim.x * WARPS32;
    unsigned long long solved = 0;
    for (long long segi = (long long)blockIdx.x * WARPS32 + warp; segi < total; segi += stride) {
        const int base = template_segment(J, P, segi, lane, delta_sm[warp]);
        __syncwarp();
        const int x0 = (int)(segi % P.nseg) * 32;
        const int cnt = min(32, J.nx - x0);
        NodeFetch next = fetch_node(J, P, base, lane);
        for (int b = 0; b < cnt; ++b) {
            const NodeFetch cur = next;
            next = fetch_node(J, P, b + 1 < cnt ? base + b + 1 : -1, lane);
            solved += exact32_node(J, P, S, cur, lane);
            __syncwarp();
        }
    }
    if (lane == 0 && solved) atomicAdd(J.n_fp64, solved);
}

constexpr size_t SMEM32 = sizeof(SysSmem) * WARPS32;

// The simulated value of one node of sequential Gaussian simulation from its
// neighbour list (`list`, `n` entries, in shared memory): the exact system,
// the estimate and variance by exact_system's and write_outputs' rules,
// and the value xp sqrt(variance) + estimate (sgs_value's rule), kept in
// registers instead of going through the status / variance / estimate
// arrays.  Written to the property and its mask by lane 0.
template <int NC, typename SM>
__device__ __forceinline__ void sgs_node32(const DevJob &J, const DevPlan &P, SM &S, int node, const int *list, int n,
                                           double xp, int lane) {
    NodeFetch f;
    f.node = node;
    f.n = n;
    f.cell = lane < n ? list[lane] : 0;
    f.cell2 = 0;
    f.informed = false;
    const NodeData d = load_node(J, P, S, f, lane);
    const bool ordinary = J.kind == 0;
    int status = ST_NO_NEIGHBOURS;
    double variance = 0.0;
    float est = 0.f;
    if (n > 0) {
        double w;
        status = exact_core<false, NC>(J, P, S, lane, d, 0.0, w);
        if (status == ST_SUCCESS) {
            double v = seq_dsum(P.c0, -__dmul_rn(w, d.b), n, S.vd, lane);
            if (ordinary) v = __dsub_rn(v, __shfl_sync(FULL_MASK, w, n - 1));
            variance = v;
            const float term = __double2float_rn(__dmul_rn(w, (double)d.dv));
            const float m0 = J.kind == 1 ? J.sk_mean_f : (J.kind == 2 ? J.mean[node] : 0.f);
            est = seq_fsum(m0, term, n, S.vf[0], lane);
        }
    }
    if (lane == 0) {
        const double value = status == ST_SUCCESS ? __dadd_rn(__dmul_rn(xp, __dsqrt_rn(variance)), (double)est)
                                                  : __dadd_rn(__dmul_rn(xp, 1.0), 0.0);
        J.sim_values[node] = __double2float_rn(value);
        J.sim_mask[node] = 1;
    }
}

// One speculative round of sequential simulation (at most 32 neighbours) for
// the jobs the tiled kernels do not take: one warp per pending node of window buffer `cur`: the template search with
// conflict detection (the list in shared memory), the exact FP64 system and
// the simulated value.
__global__ void __launch_bounds__(WARPS32 * 32) k_sgs_try32(DevJob J, DevPlan P, SgsState G, int cur) {
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    SysSmem &S = reinterpret_cast<SysSmem *>(dyn_smem)[warp];
    const int ntry = G.ctl->ntry;
    const int *win = cur ? G.win1 : G.win0;
    // the round's tries are handed out one at a time as warps free up
    int slot, rank;
    int *list = reinterpret_cast<int *>(S.row);  // 64 ints, unused by the exact path
    while (sgs_next_try(G, win, ntry, lane, slot, rank)) {
        const int node = G.nodes[rank];
        int cnt;
        const int blocker = template_node_spec(J, P, G, node, rank, lane, list, cnt);
        __syncwarp();
        if (blocker < 0) {
            sgs_node32<N32>(J, P, S, node, list, cnt, G.xp[rank], lane);
            __syncwarp();
        }
        if (lane == 0) {
            G.ok[slot] = blocker < 0;
            if (blocker >= 0) G.blocker[rank] = blocker;
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// Sequential indicator simulation (do_sis, sequential_indicator_simulation.cpp:23-116).

// Row `lane` of category k's system: dv = indicator - mean of the neighbour
// (float, combiner.h:18-22), b = C(x_lane - x0), scaled by sg sgc with the
// correlogram weights (sg: the neighbour's sigma).
template <typename SM>
__device__ __forceinline__ NodeData sis_load32(const DevJob &J, const DevPlan &P, SM &S, int node,
                                               const int *list, int n, int k, double sgc, int lane, double &sg) {
    NodeData d;
    d.n = n;
    int x0, y0, z0;
    node_xyz(J, node, x0, y0, z0);
    d.dv = 0.f;
    d.code = -1;
    d.b = 0.0;
    sg = 0.0;
    int ox = 0, oy = 0, oz = 0;
    if (lane < n) {
        const int cell = list[lane];
        int qx, qy, qz;
        node_xyz(J, cell, qx, qy, qz);
        ox = qx - x0;
        oy = qy - y0;
        oz = qz - z0;
        const float m = sis_mean(J, k, cell);
        d.dv = __fsub_rn(J.codes[cell] == k ? 1.f : 0.f, m);
        d.b = cov_at(P, ox, oy, oz, J.err);
        if (J.sis_corr) {
            sg = sis_sigma(m);
            d.b = __dmul_rn(d.b, __dmul_rn(sg, sgc));
        }
    }
    d.ox = ox;
    d.oy = oy;
    d.oz = oz;
    d.lin = oz * P.syx + oy * P.sx + ox;
    S.nb[lane] = make_int4(ox, oy, oz, d.lin);
    __syncwarp();
    return d;
}

// One speculative round of sequential indicator simulation (every category
// at most 32 neighbours) where the category groups are not solved apart: the
// correlogram weights scale each category's system by its own means.  One warp
// per pending node, the categories in
// order; per category the template search with conflict detection, the
// simple kriging system (correlogram-scaled with the mean cubes when asked)
// and the probability m_c + sum w_i (ind_i - m_i) accumulated in double
// (kriging_interpolation.h:228-265 with a double result), the mean when the
// kriging fails.  Two categories krige category 0 only and take 1 - p for
// the other (median SIS).  The code is drawn from the float probabilities.
template <int NC>
__global__ void __launch_bounds__(WARPS32 * 32) k_sis_try32(DevJob J, const DevPlan *plans, SgsState G, int cur) {
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    using SM = SysSmemN<NC * 34>;
    SM &S = reinterpret_cast<SM *>(dyn_smem)[warp];
    const int ntry = G.ctl->ntry;
    const int *win = cur ? G.win1 : G.win0;
    const int cats = J.K == 2 ? 1 : J.K;
    // the round's tries are handed out one at a time as warps free up
    int slot, rank;
    while (sgs_next_try(G, win, ntry, lane, slot, rank)) {
        const int node = G.nodes[rank];
        int *list = reinterpret_cast<int *>(S.row);  // 64 ints, unused by the exact path
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
                double sg, w;
                const NodeData d = sis_load32(J, P, S, node, list, cnt, k, sgc, lane, sg);
                const int status = J.sis_corr ? exact_core<true, NC>(J, P, S, lane, d, sg, w)
                                              : exact_core<false, NC>(J, P, S, lane, d, 0.0, w);
                if (status == ST_SUCCESS)
                    prob = seq_dsum((double)mc, __dmul_rn(w, (double)d.dv), cnt, S.vd, lane);
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

// The searches of a simulation round on their own (the systems follow in
// k_sgs_solve): one warp per tried node, which needs neither the registers
// nor the shared memory of a system, so twice the warps hide the walk's
// latency, and the finished searches' systems share warps.
__global__ void __launch_bounds__(256) k_sgs_search(DevJob J, DevPlan P, SgsState G, int cur) {
    const int lane = threadIdx.x & 31;
    const int ntry = G.ctl->ntry;
    const int *win = cur ? G.win1 : G.win0;
    // a fixed share each: handing the tries out one at a time made the round
    // wait for tens of thousands of updates of one counter
    const int warps = (int)(gridDim.x * (blockDim.x >> 5));
    for (int k = (int)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)); k < ntry; k += warps) {
        const int slot = G.trylist[k];
        const int rank = win[slot];
        const int node = G.nodes[rank];
        int cnt;
        const int blocker = template_node_spec(J, P, G, node, rank, lane, G.lists + (long long)slot * P.nmax, cnt);
        if (lane == 0) {
            G.ok[slot] = blocker < 0;
            if (blocker < 0) {
                G.counts[slot] = cnt;
                G.solvelist[atomicAdd(&G.ctl->nsolve, 1)] = slot;
            } else {
                G.blocker[rank] = blocker;
            }
        }
        __syncwarp();
    }
}

// The searches of an indicator-simulation round: a node's category groups in
// turn, until one meets a blocker.
__global__ void __launch_bounds__(256) k_sis_search(DevJob J, const DevPlan *plans, int groups, int stride, SgsState G,
                                                    int cur) {
    const int lane = threadIdx.x & 31;
    const int ntry = G.ctl->ntry;
    const int *win = cur ? G.win1 : G.win0;
    const int warps = (int)(gridDim.x * (blockDim.x >> 5));
    for (int k = (int)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)); k < ntry; k += warps) {
        const int slot = G.trylist[k];
        const int rank = win[slot];
        const int node = G.nodes[rank];
        int blocker = -1;
        for (int g = 0; g < groups && blocker < 0; ++g) {
            const long long at = (long long)slot * groups + g;
            int cnt;
            blocker = template_node_spec(J, plans[g], G, node, rank, lane, G.lists + at * stride, cnt);
            if (lane == 0) G.counts[at] = cnt;
        }
        if (lane == 0) {
            G.ok[slot] = blocker < 0;
            if (blocker < 0) G.solvelist[atomicAdd(&G.ctl->nsolve, 1)] = slot;
            else G.blocker[rank] = blocker;
        }
        __syncwarp();
    }
}

// Draws the codes of the round's solved nodes from their probabilities.
__global__ void __launch_bounds__(256) k_sis_draw(DevJob J, SgsState G, int cur) {
    const int count = G.ctl->nsolve;
    const int *win = cur ? G.win1 : G.win0;
    for (int i = blockIdx.x * 256 + threadIdx.x; i < count; i += gridDim.x * 256) {
        const int rank = win[G.solvelist[i]], node = G.nodes[rank];
        J.sim_codes[node] = (uint8_t)sis_sample(J.probs + (long long)node * J.K, J.K, G.xp[rank]);
        J.sim_mask[node] = 1;
    }
}

// A simulation's systems take every other of the solve's tiles (launch_solve32):
// a round's solve is the smaller part of it beside the search, and 24 in place
// of 20 and 32 in place of 28 cost SGS 166x141x100 20.24 for 19.47 ms and 30.5
// for 29.5.  Above 32 neighbours search and system stay in one warp
// (launch_sgs_try64), 131 ms at 40 and 218 at 64 there; the tiles of up to 64
// in a trial build took 48 and 114.
bool sim_tiles(const DevPlan &P) { return P.nmax <= 32 && tile_takes(P); }

void launch_sis_groups(const DevJob &J, const SisGroups &groups, const SgsState &G, int cur, cudaStream_t s) {
    const long long g = persistent_grid((const void *)k_sis_search, 256, 0, 0, 1LL << 30);
    k_sis_search<<<(unsigned)g, 256, 0, s>>>(J, groups.dev, groups.n, groups.stride, G, cur);
    for (int i = 0; i < groups.n; ++i) {
        const SisGroup &q = groups.groups[i];
        const int st = groups.stride, n = groups.n, m = q.plan.nmax;
        // the solve list is handed out once per group (the commit resets it)
        if (i > 0) cudaMemsetAsync(&G.ctl->solve_cursor, 0, sizeof(unsigned), s);
        if (m <= 8) launch_sis_solve<TileGeom<8, 4, 1, 2, 10>, 4, 5>(J, q.plan, G, cur, st, n, i, q.k0, q.k1, s);
        else if (m <= 12) launch_sis_solve<TileGeom<12, 4, 1, 4, 10>, 4, 4>(J, q.plan, G, cur, st, n, i, q.k0, q.k1, s);
        else if (m <= 16) launch_sis_solve<TileGeom<16, 4, 1, 2, 10>, 4, 3>(J, q.plan, G, cur, st, n, i, q.k0, q.k1, s);
        else if (m <= 24) launch_sis_solve<TileGeom<24, 4, 1, 2, 10>, 4, 2>(J, q.plan, G, cur, st, n, i, q.k0, q.k1, s);
        else launch_sis_solve<TileGeom<32, 4, 2, 4, 8>, 4, 2>(J, q.plan, G, cur, st, n, i, q.k0, q.k1, s);
    }
    k_sis_draw<<<(unsigned)(g < 592 ? g : 592), 256, 0, s>>>(J, G, cur);
}

void launch_sgs_try32(const DevJob &J, const DevPlan &P, const SgsState &G, int cur, cudaStream_t s) {
    if (G.lists) {
        const long long g = persistent_grid((const void *)k_sgs_search, 256, 0, 0, 1LL << 30);
        k_sgs_search<<<(unsigned)g, 256, 0, s>>>(J, P, G, cur);
        if (P.nmax <= 8) launch_sgs_solve<TileGeom<8, 4, 1, 2, 10>, 4, 5>(J, P, G, cur, s);
        else if (P.nmax <= 12) launch_sgs_solve<TileGeom<12, 4, 1, 4, 10>, 4, 4>(J, P, G, cur, s);
        else if (P.nmax <= 16) launch_sgs_solve<TileGeom<16, 4, 1, 2, 10>, 4, 3>(J, P, G, cur, s);
        else if (P.nmax <= 24) launch_sgs_solve<TileGeom<24, 4, 1, 2, 10>, 4, 2>(J, P, G, cur, s);
        else launch_sgs_solve<TileGeom<32, 4, 2, 4, 8>, 4, 2>(J, P, G, cur, s);
        return;
    }
    const long long g = persistent_grid((const void *)k_sgs_try32, WARPS32 * 32, SMEM32, 0, 1LL << 30);
    k_sgs_try32<<<(unsigned)g, WARPS32 * 32, SMEM32, s>>>(J, P, G, cur);
}

void launch_sis_try32(const DevJob &J, const DevPlan *plans, const SgsState &G, int cur, cudaStream_t s) {
    if (J.nb_stride <= N16) {
        constexpr size_t smem = sizeof(SysSmem16) * WARPS32;
        const long long g = persistent_grid((const void *)k_sis_try32<N16>, WARPS32 * 32, smem, 0, 1LL << 30);
        k_sis_try32<N16><<<(unsigned)g, WARPS32 * 32, smem, s>>>(J, plans, G, cur);
        return;
    }
    const long long g = persistent_grid((const void *)k_sis_try32<N32>, WARPS32 * 32, SMEM32, 0, 1LL << 30);
    k_sis_try32<N32><<<(unsigned)g, WARPS32 * 32, SMEM32, s>>>(J, plans, G, cur);
}

void launch_fused32(const DevJob &J, const DevPlan &P, cudaStream_t s, int blocks_per_sm) {
    const long long segs = (long long)P.nseg * J.ny * J.nz;
    if (segs <= 0) return;
    const int threads = WARPS32 * 32;
    const long long g =
        persistent_grid((const void *)k_fused32, threads, SMEM32, blocks_per_sm, (segs + WARPS32 - 1) / WARPS32);
    k_fused32<<<(unsigned)g, threads, SMEM32, s>>>(J, P);
}

// The tile of a job's systems by its largest neighbour count.  Fewer lanes a
// system share each step's pivot chain among more systems and read fewer
// shared-memory words per product, until the lane's accumulators no longer
// fit the registers: 4 lanes (8 systems a warp) up to 24 neighbours, 8 above;
// the panel (row blocks whose sums are kept open together) trades spilled
// registers, which every width has some of, for passes over the finished rows.
// Panels of another width on SK 256x256x64 with the neighbour count set, in ms
// (panel taken [width: ms]): 12: 2.01 [2: 1.95]   16: 3.20 [4: 3.28]   20: 7.25
// [4: 6.42]   24: 9.65 [4: 9.33]   28: 14.8 [2: 17.0, 6: 15.4]   32: 17.4 [2:
// 17.6, 6: 18.6]; up to 24 the other width spills more (24: 300 bytes for 8)
// and is the faster one at 12, 20 and 24 all the same.  Solve of the IK 200x200x100 job (4.0 M systems) with
// the neighbour count set, in ms:
//   8: 1.06   12: 1.99   16: 3.09   20: 7.1   24: 9.1   28: 14.5
// against 39.7 at 24 with one column per lane and one system a warp; SK
// 256x256x64 (4.15 M systems, 32 neighbours) 17.5 against 53.2, OK 19.7
// against 57.1.  The neighbouring tiles, measured on earlier builds: 12 as 8
// lanes 3.5; 16 as 8 lanes 5.2; 20 as 8 lanes 8.4; 24 as 8 lanes 9.6; 32 as
// 16 lanes 21.0 where 8 lanes took 19.2.
void launch_solve32(const DevJob &J, const DevPlan &P, cudaStream_t s, int blocks_per_sm) {
    const int b = blocks_per_sm;
    if (!tile_takes(P)) {
        const long long g = persistent_grid((const void *)k_solve_exact32, WARPS32 * 32, SMEM32, b,
                                            (J.size + WARPS32 - 1) / WARPS32);
        k_solve_exact32<<<(unsigned)g, WARPS32 * 32, SMEM32, s>>>(J, P);
    } else if (P.nmax <= 8) {
        launch_tile<TileGeom<8, 4, 1, 2, 10>, 4, 5>(J, P, s, b);
    } else if (P.nmax <= 12) {
        launch_tile<TileGeom<12, 4, 1, 4, 10>, 4, 4>(J, P, s, b);
    } else if (P.nmax <= 16) {
        launch_tile<TileGeom<16, 4, 1, 2, 10>, 4, 3>(J, P, s, b);
    } else if (P.nmax <= 20) {
        launch_tile<TileGeom<20, 4, 1, 2, 10>, 4, 2>(J, P, s, b);
    } else if (P.nmax <= 24) {
        launch_tile<TileGeom<24, 4, 1, 2, 10>, 4, 2>(J, P, s, b);
    } else if (P.nmax <= 28) {
        launch_tile<TileGeom<28, 4, 2, 4, 8>, 4, 2>(J, P, s, b);
    } else {
        launch_tile<TileGeom<32, 4, 2, 4, 8>, 4, 2>(J, P, s, b);
    }
}

}  // namespace hpgl_b200
