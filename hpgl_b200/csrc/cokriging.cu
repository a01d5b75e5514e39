// Colocated simple cokriging, Markov models I and II
// (simple_cokriging_markI.cpp:19-307), FP64 in the reference's exact operation
// order: several systems a warp on lane tiles (cok_tile.cuh), and one warp per
// node (this file's k_cokriging) for more than 48 neighbours and for the nodes
// whose elimination needs the search for a pivot row.
//
// The neighbours come from the template search (neighbour_lookup_t over the
// untruncated primary model; the reference uses no clusterizer here).  The
// (N+1)-row system -- primary covariances, the cross covariances
// coef * C_x(center - x_i) in its last row and column, the secondary variance
// in the corner -- is solved by the reference's gauss_solve
// (gauss_solver.cpp:5-63): for column i the first row not yet used whose
// entry is non-zero is the pivot row, it is divided by its pivot entry (here
// with the correctly rounded reciprocal and one fused correction, which is
// the IEEE quotient), and eliminated from every unused row; the back
// substitution starts each unknown from B at its own position (B[i], as the
// reference does) and subtracts the pivot rows' terms from the last column
// down.  In k_cokriging the system lives row-major in shared memory; lane l
// owns rows l, l + 32 and l + 64 (the last only for lane 0).
#include <algorithm>

#include "cok_tile.cuh"
#include "device_common.cuh"

namespace hpgl_b200 {

namespace {


// The shared area of one warp, sized for the job's largest system (rows =
// max_neighbours + 1): the row-major system with an odd row stride (the
// lanes' own-row accesses spread over the banks), B, the neighbour offsets
// and the pivot order.
struct CokSmem {
    double *A;
    double *B;
    int4 *nb;
    int *order;
    int ld;
};

__host__ __device__ inline int cok_ld(int nmax) { return (nmax + 1) | 1; }
__host__ __device__ inline size_t cok_smem_bytes(int nmax) {
    const int rows = nmax + 1, ld = cok_ld(nmax);
    return (size_t)rows * ld * 8 + (size_t)rows * 8 + 64 * 16 + (size_t)rows * 4 + 16;
}

__device__ __noinline__ double crcp(double a) { return __drcp_rn(a); }

// Value of position i (0..64) held by lane i % 32 in slot i / 32.
__device__ __forceinline__ double slot_val(double v0, double v1, double v2, int i) {
    const double v = i < 32 ? v0 : (i < 64 ? v1 : v2);
    return __shfl_sync(FULL_MASK, v, i & 31);
}

__device__ void cok_node(const DevJob &J, const DevPlan &P, CokSmem &S, int node, int lane,
                         unsigned long long &solved) {
    const long long slot = node;
    const int LD = S.ld;
    const float m1 = J.cok_m1, m2 = J.cok_m2;
    if (J.mask[node]) {
        // informed primary: copied (set_at, simple_cokriging_markI.cpp:245-248)
        if (lane == 0) {
            J.out_values[node] = J.values[node];
            J.out_mask[node] = 1;
            J.status[slot] = ST_NOT_KRIGED;
        }
        return;
    }
    const float sv = J.smask[node] ? J.svalues[node] : m2;
    const int n = J.nbcount[node];
    const int ms = n + 1;
    int status = ST_NO_NEIGHBOURS;
    float result = 0.f;
    double w0 = 0.0, w1 = 0.0, w2 = 0.0;
    if (n > 0) {
        int x0, y0, z0;
        node_xyz(J, node, x0, y0, z0);
        float v0 = 0.f, v1 = 0.f;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r = lane + 32 * h;
            int4 o = make_int4(0, 0, 0, 0);
            if (r < n) {
                const int cell = J.nb[(long long)node * P.nmax + r];
                int qx, qy, qz;
                node_xyz(J, cell, qx, qy, qz);
                o = make_int4(qx - x0, qy - y0, qz - z0, 0);
                o.w = o.z * P.syx + o.y * P.sx + o.x;
                (h ? v1 : v0) = J.values[cell];
            }
            S.nb[r] = o;
        }
        __syncwarp();
        // build_system (simple_cokriging_markI.cpp:19-54): A(i,k) = C(x_i - x_k)
        // for i != k < n; the table is exactly symmetric (C(v) = C(-v) bit for
        // bit), so either orientation gives the reference's value.  Pairs
        // (r, r + d) along cyclic diagonals, all of a lane's gathers of a trip
        // in flight: for n <= 32, lane l takes (l, l+d mod 32), d = 1..16 (d = 16
        // on lanes 0-15 only); above, the pairs of its rows l and l+32 with
        // d = 1..31 mod 64 and (l, l+32).
        if (n <= 32) {
            const int4 a = S.nb[lane];
            double v[16];
#pragma unroll
            for (int d = 1; d <= 16; ++d) {
                const int k = (lane + d) & 31;
                v[d - 1] = 0.0;
                if (lane < n && k < n && (d < 16 || lane < 16)) {
                    const int4 c = S.nb[k];
                    v[d - 1] = cov_lin(P, a.x - c.x, a.y - c.y, a.z - c.z, a.w - c.w, J.err);
                }
            }
#pragma unroll
            for (int d = 1; d <= 16; ++d) {
                const int k = (lane + d) & 31;
                if (lane < n && k < n && (d < 16 || lane < 16)) {
                    S.A[lane * LD + k] = v[d - 1];
                    S.A[k * LD + lane] = v[d - 1];
                }
            }
        } else {
            const int4 own[2] = {S.nb[lane], S.nb[lane + 32]};
#pragma unroll 1
            for (int d0 = 1; d0 <= 32; d0 += 8) {
                double v[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    const int d = d0 + (e >> 1), h = e & 1;
                    const int r = lane + 32 * h, k = (r + d) & 63;
                    v[e] = 0.0;
                    if (r < n && k < n && (d < 32 || h == 0)) {
                        const int4 c = S.nb[k];
                        v[e] = cov_lin(P, own[h].x - c.x, own[h].y - c.y, own[h].z - c.z, own[h].w - c.w, J.err);
                    }
                }
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    const int d = d0 + (e >> 1), h = e & 1;
                    const int r = lane + 32 * h, k = (r + d) & 63;
                    if (r < n && k < n && (d < 32 || h == 0)) {
                        S.A[r * LD + k] = v[e];
                        S.A[k * LD + r] = v[e];
                    }
                }
            }
        }
        const double c0 = __ldg(P.table);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r = lane + 32 * h;
            if (r < n) {
                const int4 a = S.nb[r];
                S.A[r * LD + r] = c0;
                // cross_cov(center, x_r) = coef * C_x(center - x_r); C_x(-v) = C_x(v)
                double cx = 0.0;
                if (cov_in_range(P, a.x, a.y, a.z)) cx = __ldg(J.cross_table + abs(a.w));
                else if (!P.truncated) atomicOr(J.err, DERR_TABLE_RANGE);
                const double x = __dmul_rn(J.cok_coef, cx);
                S.A[n * LD + r] = x;
                S.A[r * LD + n] = x;
                S.B[r] = cov_lin(P, a.x, a.y, a.z, a.w, J.err);  // primary_cov(x_r, center)
            }
        }
        if (lane == 0) {
            S.B[n] = __dmul_rn(J.cok_coef, __ldg(J.cross_table));
            S.A[n * LD + n] = J.cok_svar;
        }
        __syncwarp();
        // gauss_solve (gauss_solver.cpp:5-63)
        bool used0 = false, used1 = false, used2 = false;  // flags of the lane's rows
        bool singular = false;
        for (int i = 0; i < ms; ++i) {
            const int r0 = lane, r1 = lane + 32, r2 = lane + 64;
            const bool c0ok = r0 < ms && !used0 && S.A[r0 * LD + i] != 0.0;
            const bool c1ok = r1 < ms && !used1 && S.A[r1 * LD + i] != 0.0;
            const bool c2ok = r2 < ms && !used2 && S.A[r2 * LD + i] != 0.0;
            const unsigned b0 = __ballot_sync(FULL_MASK, c0ok), b1 = __ballot_sync(FULL_MASK, c1ok),
                           b2 = __ballot_sync(FULL_MASK, c2ok);
            int row;
            if (b0) row = __ffs(b0) - 1;
            else if (b1) row = 32 + __ffs(b1) - 1;
            else if (b2) row = 64 + __ffs(b2) - 1;
            else {
                singular = true;
                break;
            }
            if (row == r0) used0 = true;
            if (row == r1) used1 = true;
            if (row == r2) used2 = true;
            if (lane == 0) S.order[i] = row;
            const double coef = S.A[row * LD + i];
            const double y = crcp(coef);
            __syncwarp();
            // normalise the pivot row from column i on, and its B
            for (int j = i + lane; j < ms; j += 32) S.A[row * LD + j] = div_by_rcp(S.A[row * LD + j], coef, y);
            if (lane == 0) S.B[row] = div_by_rcp(S.B[row], coef, y);
            __syncwarp();
            // eliminate column i from every unused row.  The unused rows are
            // listed (in shared memory; the neighbour offsets are no longer
            // needed) and dealt out to the lanes in turn, so that no lane
            // takes two rows while another is idle (a 33-row system would
            // otherwise leave lane 0 two rows per step).
            const double *pr = S.A + row * LD;
            const double bp = S.B[row];
            int *live = reinterpret_cast<int *>(S.nb);
            const bool l0 = lane < ms && !used0, l1 = lane + 32 < ms && !used1, l2 = lane + 64 < ms && !used2;
            const unsigned lb0 = __ballot_sync(FULL_MASK, l0), lb1 = __ballot_sync(FULL_MASK, l1),
                           lb2 = __ballot_sync(FULL_MASK, l2);
            const unsigned below = (1u << lane) - 1u;
            if (l0) live[__popc(lb0 & below)] = lane;
            if (l1) live[__popc(lb0) + __popc(lb1 & below)] = lane + 32;
            if (l2) live[__popc(lb0) + __popc(lb1) + __popc(lb2 & below)] = lane + 64;
            const int nlive = __popc(lb0) + __popc(lb1) + __popc(lb2);
            __syncwarp();
            for (int t = lane; t < nlive; t += 32) {
                const int r = live[t];
                double *ar = S.A + r * LD;
                const double c = ar[i];
                for (int k = i; k < ms; ++k) ar[k] = __dsub_rn(ar[k], __dmul_rn(c, pr[k]));
                S.B[r] = __dsub_rn(S.B[r], __dmul_rn(c, bp));
            }
            __syncwarp();
        }
        if (!singular) {
            // back substitution: X[i] = B[i] - sum_{j>i, j descending} A[order[i]][j] X[j]
            double x0 = lane < ms ? S.B[lane] : 0.0;
            double x1 = lane + 32 < ms ? S.B[lane + 32] : 0.0;
            double x2 = lane + 64 < ms ? S.B[lane + 64] : 0.0;
            const int o0 = lane < ms ? S.order[lane] : 0;
            const int o1 = lane + 32 < ms ? S.order[lane + 32] : 0;
            const int o2 = lane + 64 < ms ? S.order[lane + 64] : 0;
            for (int j = ms - 1; j > 0; --j) {
                const double xj = slot_val(x0, x1, x2, j);
                if (lane < j) x0 = __dsub_rn(x0, __dmul_rn(S.A[o0 * LD + j], xj));
                if (lane + 32 < j) x1 = __dsub_rn(x1, __dmul_rn(S.A[o1 * LD + j], xj));
                if (lane + 64 < j) x2 = __dsub_rn(x2, __dmul_rn(S.A[o2 * LD + j], xj));
            }
            w0 = x0;
            w1 = x1;
            w2 = x2;
            // combine (simple_cokriging_markI.cpp:84-105): float result, each
            // step widened to double and rounded back
            const float t0 = __fsub_rn(v0, m1), t1 = __fsub_rn(v1, m1);
            float res = m1;
            for (int i = 0; i < n; ++i) {
                const float ti = __shfl_sync(FULL_MASK, i < 32 ? t0 : t1, i & 31);
                const double wi = slot_val(w0, w1, w2, i);
                res = __double2float_rn(__dadd_rn((double)res, __dmul_rn((double)ti, wi)));
            }
            const double wn = slot_val(w0, w1, w2, n);
            res = __double2float_rn(__dadd_rn((double)res, __dmul_rn(wn, (double)__fsub_rn(sv, m2))));
            result = res;
            status = ST_SUCCESS;
        } else {
            status = ST_SINGULAR;
        }
        ++solved;
    }
    if (status != ST_SUCCESS) result = __fsub_rn(__fadd_rn(m1, sv), m2);  // failure estimate
    if (lane == 0) {
        J.out_values[node] = result;
        J.out_mask[node] = 1;
        J.status[slot] = (int8_t)status;
    }
    if (J.weights && status == ST_SUCCESS) {
        double *wdst = J.weights + slot * (P.nmax + 1);
        if (lane < ms) wdst[lane] = w0;
        if (lane + 32 < ms) wdst[lane + 32] = w1;
        if (lane + 64 < ms) wdst[lane + 64] = w2;
    }
}

// redo: the nodes the tiled kernel marked; else every node.
__global__ void __launch_bounds__(32) k_cokriging(DevJob J, DevPlan P, bool redo) {
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    CokSmem S;
    {
        const int rows = P.nmax + 1;
        S.ld = cok_ld(P.nmax);
        S.nb = reinterpret_cast<int4 *>(dyn_smem);  // 16-byte aligned first
        S.A = reinterpret_cast<double *>(dyn_smem + 64 * 16);
        S.B = S.A + (size_t)rows * S.ld;
        S.order = reinterpret_cast<int *>(S.B + rows);
    }
    const int lane = threadIdx.x & 31;
    unsigned long long solved = 0;
    if (redo) {
        for (long long base = (long long)blockIdx.x * 32; base < J.size; base += (long long)gridDim.x * 32) {
            const long long i = base + lane;
            unsigned m = __ballot_sync(FULL_MASK, i < J.size && J.status[i] == COK_REDO);
            while (m) {
                const int k = __ffs(m) - 1;
                m &= m - 1;
                cok_node(J, P, S, (int)(base + k), lane, solved);
                __syncwarp();
            }
        }
    } else {
        for (long long node = blockIdx.x; node < J.size; node += gridDim.x) {
            cok_node(J, P, S, (int)node, lane, solved);
            __syncwarp();
        }
    }
    if (lane == 0 && solved) atomicAdd(J.n_fp64, solved);
}

}  // namespace

static void launch_general(const DevJob &J, const DevPlan &P, bool redo, cudaStream_t s) {
    // the occupancy lookup is cached per kernel: ask it for the largest area,
    // and size this grid from the job's own area
    const size_t smem = cok_smem_bytes(P.nmax);
    const long long cap = persistent_grid((const void *)k_cokriging, 32, cok_smem_bytes(64), 0, J.size);
    int per_sm = 0, dev = 0, sms = 148;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_cokriging, 32, smem);
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    long long g = (long long)std::max(1, per_sm) * sms;
    g = std::max<long long>(cap, std::min<long long>(g, J.size));
    if (redo) g = std::min<long long>(g, (J.size + 31) / 32);
    k_cokriging<<<(unsigned)g, 32, smem, s>>>(J, P, redo);
}

template <typename T, int WARPS, int MINB>
static void launch_cok_tile(const DevJob &J, const DevPlan &P, cudaStream_t s) {
    constexpr size_t smem = sizeof(double) * T::SIZE * T::G * WARPS;
    const long long units = (J.size + WARPS * T::G - 1) / (WARPS * T::G);
    const long long g = persistent_grid((const void *)k_cok_tile<T, WARPS, MINB>, WARPS * 32, smem, 0, units);
    k_cok_tile<T, WARPS, MINB><<<(unsigned)g, WARPS * 32, smem, s>>>(J, P);
    launch_general(J, P, true, s);
}

// The tile of a job's systems by its largest neighbour count: as many lanes a
// system as the square takes to fit the registers (4 lanes up to 12
// neighbours, 8 up to 24, 16 up to 36, a whole warp up to 48).  Elimination of
// 0.88 M systems (161x119x47) in ms, in brackets one system a warp with a row
// per lane in shared memory:
//   8: 0.44 [4.5]   12: 0.82 [6.5]   16: 1.76 [8.8]   20: 3.06 [11.2]
//   24: 4.46 [13.7]   28: 6.65 [16.5]   36: 11.5 [26.4]   40: 17.0 [32.3]
//   44: 19.7 [38.5]   48: 28.8 [52.6]
// and of 4.11 M (256x256x64): 32: 37.5 [90.9].  Neighbouring tiles: 12 as 8
// lanes 1.09, 16 as 16 lanes 2.29, 24 as 16 lanes 4.61, 32 as a whole warp
// 47.8, 36 as a whole warp 13.6.  Above 48 the square no longer fits a warp's
// registers.
void launch_cokriging(const DevJob &J, const DevPlan &P, cudaStream_t s) {
    if (J.size <= 0) return;
    if (!cok_tile_takes(P)) launch_general(J, P, false, s);
    else if (P.nmax <= 8) launch_cok_tile<CokGeom<8, 4, 1>, 4, 4>(J, P, s);
    else if (P.nmax <= 12) launch_cok_tile<CokGeom<12, 4, 1>, 4, 3>(J, P, s);
    else if (P.nmax <= 16) launch_cok_tile<CokGeom<16, 4, 2>, 4, 3>(J, P, s);
    else if (P.nmax <= 20) launch_cok_tile<CokGeom<20, 4, 2>, 4, 2>(J, P, s);
    else if (P.nmax <= 24) launch_cok_tile<CokGeom<24, 4, 2>, 1, 7>(J, P, s);
    else if (P.nmax <= 28) launch_cok_tile<CokGeom<28, 4, 4>, 1, 10>(J, P, s);
    else if (P.nmax <= 32) launch_cok_tile<CokGeom<32, 4, 4>, 1, 8>(J, P, s);
    else if (P.nmax <= 36) launch_cok_tile<CokGeom<36, 4, 4>, 1, 7>(J, P, s);
    else if (P.nmax <= 40) launch_cok_tile<CokGeom<40, 8, 4>, 1, 10>(J, P, s);
    else if (P.nmax <= 44) launch_cok_tile<CokGeom<44, 8, 4>, 1, 8>(J, P, s);
    else launch_cok_tile<CokGeom<48, 8, 4>, 1, 8>(J, P, s);
}

}  // namespace hpgl_b200
