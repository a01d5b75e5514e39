// CUDA kernels of the kriging pipeline for sm_100a (the per-node solves are
// in solve32.cu and solve64.cu):
//   k_build_bits       informed mask -> padded bit rows
//   k_search_template  bit-sliced walk of the sorted search template
//   k_search_cluster   clusterizer gather, covariance filter, reference sort
//   k_ik_argmax        most probable category
//   k_sgs_*            bookkeeping of the speculative simulation rounds
// Paths cited are relative to the reference's src/geo_bsd/hpgl/.
#include <algorithm>
#include <climits>
#include <cstdio>
#include <map>
#include <mutex>

#include "device_common.cuh"
#include "introsort.h"
#include "search_common.cuh"
#include "kernels.cuh"

namespace hpgl_b200 {

// ---------------------------------------------------------------------------
// informed-bit rows: bit j of word w of row (z*ny + y) is padded x = 32w + j,
// i.e. grid x = 32w + j - px.
__global__ void k_build_bits(DevJob J, DevPlan P, uint32_t *bits) {
    long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    long long rows = (long long)J.ny * J.nz;
    if (t >= rows * P.wpr) return;
    long long row = t / P.wpr;
    int w = (int)(t % P.wpr);
    uint32_t word = 0;
    const uint8_t *m = J.mask + row * J.nx;
    for (int j = 0; j < 32; ++j) {
        int x = 32 * w + j - P.px;
        if (x >= 0 && x < J.nx && m[x]) word |= 1u << j;
    }
    bits[t] = word;
}

// ---------------------------------------------------------------------------
// Template search: one warp per 32-node x-segment (template_segment in
// search_common.cuh), persistent: each warp takes the next segment from a
// counter, so warps whose segments end early (dense regions) take more and
// none waits on a fixed share at the end.
__global__ void __launch_bounds__(256) k_search_template(DevJob J, DevPlan P) {
    __shared__ int delta_sm[8][32];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const long long total = (long long)P.nseg * J.ny * J.nz;
    while (true) {
        int segi = 0;
        if (lane == 0) segi = atomicAdd(J.seg_next, 1);
        segi = __shfl_sync(FULL_MASK, segi, 0);
        if (chunk_first(segi, total) >= total) break;
        template_segment(J, P, segi, lane, delta_sm[wib]);
    }
}

// ---------------------------------------------------------------------------
// Warp form of the reference sort's partition (sort_partition_pairs): each
// round collects the next 32 left stoppers and 32 right stoppers with
// ballots, lane k holds the pair (L_k, R_k), the pairs with L_k < R_k (a
// prefix of the lanes) swap at once, and the first failing pair gives the
// cut.  Each round scans left from L_{b-1}+1 up to R_{b-1} and right from
// R_{b-1}-1 down to L_{b-1}; earlier rounds' swaps only ever turn positions
// at or beyond those bounds into stoppers, which yields the same
// min(L_m, R_{m-1}).  A range of up to 64 elements is one round of two
// elements a lane (warp_partition64).
constexpr int SORT_STACK = 72;
constexpr int TAIL_MAX = 64 + 16;        // positions the final insertion sort reaches
constexpr int SORT_BUF = TAIL_MAX + 32;  // doubles of scratch a warp

// sort_partition of [pivot + 1, hi), hi - pivot <= 64, pivot the element
// before the range: the stoppers' ranks come from two 64-bit masks, their
// positions by rank through lbuf / rbuf (64 each).
__device__ int warp_partition64(SortArr &a, int pivot, int hi, int *lbuf, int *rbuf, int lane) {
    const int m = hi - pivot;  // positions pivot + 0 (the pivot) .. pivot + m - 1
    const double pk = a.key[pivot];
    bool lst[2], rst[2];
    unsigned lb[2], rb[2];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        const int e = lane + 32 * t;
        const double k = e < m ? a.key[pivot + e] : 0.0;
        lst[t] = e > 0 && e < m && !(k > pk);
        rst[t] = e < m && !(pk > k);
        lb[t] = __ballot_sync(FULL_MASK, lst[t]);
        rb[t] = __ballot_sync(FULL_MASK, rst[t]);
    }
    const unsigned below = (1u << lane) - 1, above = ~below & ~(1u << lane);
    const int nl = __popc(lb[0]) + __popc(lb[1]), nr = __popc(rb[0]) + __popc(rb[1]);
    if (lst[0]) lbuf[__popc(lb[0] & below)] = pivot + lane;
    if (lst[1]) lbuf[__popc(lb[0]) + __popc(lb[1] & below)] = pivot + lane + 32;
    if (rst[0]) rbuf[__popc(rb[1]) + __popc(rb[0] & above)] = pivot + lane;
    if (rst[1]) rbuf[__popc(rb[1] & above)] = pivot + lane + 32;
    __syncwarp();
    int pairs = 0;
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        const int e = lane + 32 * t;
        const bool pair = e < nl && e < nr && lbuf[e] < rbuf[e];  // a prefix of the ranks
        if (pair) a.swap(lbuf[e], rbuf[e]);
        pairs += __popc(__ballot_sync(FULL_MASK, pair));
    }
    const int lm = pairs < nl ? lbuf[pairs] : INT_MAX, rm = pairs > 0 ? rbuf[pairs - 1] : INT_MAX;
    __syncwarp();
    return lm < rm ? lm : rm;
}

__device__ int warp_partition(SortArr &a, int lo, int hi, int pivot, int *lbuf, int *rbuf, int lane) {
    const double pk = a.key[pivot];
    const uint32_t below = (1u << lane) - 1;
    int lp = lo, lend = hi - 1;      // left scan window [lp, lend], upwards
    int rp = hi - 1, rend = pivot;   // right scan window [rend, rp], downwards
    int rprev = INT_MAX;             // R_{b-1}
    while (true) {
        int cnt = 0;
        for (int p0 = lp; cnt < 32 && p0 <= lend; p0 += 32) {
            const int p = p0 + lane;
            const bool st = p <= lend && !(a.key[p] > pk);
            const uint32_t bal = __ballot_sync(FULL_MASK, st);
            const int r = cnt + __popc(bal & below);
            if (st && r < 32) lbuf[r] = p;
            cnt += __popc(bal);
        }
        __syncwarp();
        const int my_l = lane < cnt ? lbuf[lane] : INT_MAX;
        cnt = 0;
        for (int q0 = rp; cnt < 32 && q0 >= rend; q0 -= 32) {
            const int q = q0 - lane;
            const bool st = q >= rend && !(pk > a.key[q]);
            const uint32_t bal = __ballot_sync(FULL_MASK, st);
            const int r = cnt + __popc(bal & below);
            if (st && r < 32) rbuf[r] = q;
            cnt += __popc(bal);
        }
        __syncwarp();
        const int my_r = lane < cnt ? rbuf[lane] : INT_MIN;
        const bool pair = my_l < my_r;
        const int m = __popc(__ballot_sync(FULL_MASK, pair));
        if (pair) a.swap(my_l, my_r);
        __syncwarp();
        if (m < 32) {
            const int lm = __shfl_sync(FULL_MASK, my_l, m);
            const int rl = __shfl_sync(FULL_MASK, my_r, (m + 31) & 31);
            const int rm = m > 0 ? rl : rprev;
            return lm < rm ? lm : rm;
        }
        const int l31 = __shfl_sync(FULL_MASK, my_l, 31), r31 = __shfl_sync(FULL_MASK, my_r, 31);
        lp = l31 + 1;
        lend = r31;
        rp = r31 - 1;
        rend = l31;
        rprev = r31;
    }
}

struct SortFrame {
    int lo, hi, depth;
};

// The partitioning half of reference_sort_prefix driven by a whole warp:
// control flow is uniform, lane 0 does the median-of-three and heap sorts, the
// warp the partitions.  Afterwards every position below k lies in a part of
// at most 16 elements, or in a sorted one, as the reference's sort leaves it
// for its final insertion sort.  `stack` holds SORT_STACK frames, `lbuf` and
// `rbuf` 64 positions each (shared memory).
__device__ bool warp_reference_parts(SortArr &a, int n, int k, int lane, SortFrame *stack, int *lbuf, int *rbuf) {
    if (n <= 16) return true;
    if (k > n) k = n;
    int sp = 0;
    if (lane == 0) stack[0] = SortFrame{0, n, 2 * sort_floor_log2(n)};
    ++sp;
    while (sp > 0) {
        __syncwarp();
        const SortFrame f = stack[--sp];
        int lo = f.lo, hi = f.hi, depth = f.depth;
        if (lo >= k) continue;
        while (hi - lo > 16) {
            if (depth == 0) {
                if (lane == 0) sort_heapsort(a, lo, hi);
                break;
            }
            --depth;
            const int mid = lo + (hi - lo) / 2;
            if (lane == 0) sort_median_to_first(a, lo, lo + 1, mid, hi - 1);
            __syncwarp();
            const int cut = hi - lo <= 64 ? warp_partition64(a, lo, hi, lbuf, rbuf, lane)
                                          : warp_partition(a, lo + 1, hi, lo, lbuf, rbuf, lane);
            if (cut < k) {
                if (sp >= SORT_STACK) return false;
                __syncwarp();
                if (lane == 0) stack[sp] = SortFrame{cut, hi, depth};
                ++sp;
            }
            hi = cut;
        }
    }
    __syncwarp();
    return true;
}

// The final insertion sort of reference_sort_prefix and the first k indices of
// its result, in `out`.  An insertion sort is stable and here moves elements
// within their part of at most 16 only, so the place of position i is i, plus
// the later elements before it, less the earlier elements it is before, among
// its 15 neighbours on either side: counted for 32 positions at once where
// lane 0 moved them one after another.  s: SORT_BUF doubles.
__device__ void warp_sort_tail(const SortArr &a, int n, int k, double *s, int *out, int lane) {
    const int end = k + 16 < n ? k + 16 : n;
    for (int i = lane; i < end + 32; i += 32) {
        // 16 sentinels either side: never before, never after
        double v = i < 16 ? __longlong_as_double(0x7ff0000000000000LL) : __longlong_as_double(0xfff0000000000000LL);
        if (i >= 16 && i < end + 16) v = a.key[i - 16];
        s[i] = v;
    }
    __syncwarp();
    for (int i = lane; i < end; i += 32) {
        const double v = s[i + 16];
        int at = i;
#pragma unroll 5
        for (int d = 1; d < 16; ++d) {
            if (s[i + 16 + d] > v) ++at;
            if (s[i + 16 - d] < v) --at;
        }
        if (at < k && at < n) out[at] = a.idx[i];
    }
    __syncwarp();
}

// ---------------------------------------------------------------------------
// Clusterizer search (sugarbox_indexed_neighbour_lookup.h:72-121): one warp
// per node whose 27 boxes are all within their fill limit.  The warp gathers
// the boxes' informed nodes in the reference's k-j-i / insertion order,
// keeps those with covariance above C(0)/100 (order-preserving ballot
// compaction), then the warp orders them exactly as the reference's
// std::sort does — as far as the first max_neighbours positions, which become
// the list.  Bound by instruction issue and the latency of the candidates'
// scratch (L1, L2): parts of up to 64 elements and the final insertion sort
// were lane 0's, a chain of dependent accesses each; as warp-wide counts and
// ballots LVM 512x512x32 searches in 24.4 ms (35.0), OK 61x64x12 with 60
// neighbours in 0.40 (1.32), OK 88x88x20 with 2 900 candidates a node, where
// the long partitions remain, in 8.7 (10.0).  Where most candidates of the 27
// boxes fail the filter their reads of the table are the traffic: those beyond
// the model's reach are dropped by their offset (OK 251x213x51, 13 600
// candidates of which 3 400 pass: 316 -> 274 ms), and the next candidates are
// read a chunk ahead (258).  LVM's truncated model, whose range test drops
// most anyway, pays 0.5 ms for it.
constexpr int CLUSTER_WARPS = 4;
// |reach_t d|^2 (Plan): beyond reach_limit the covariance is at most C(0)/100.
__device__ __forceinline__ float reach2(const DevPlan &P, float dx, float dy, float dz) {
    float q = 0.f;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const float u = P.reach_t[3 * i] * dx + P.reach_t[3 * i + 1] * dy + P.reach_t[3 * i + 2] * dz;
        q += u * u;
    }
    return q;
}
// Nodes a warp takes from the counter at a time: at most this many, fewer where
// a small grid would leave warps without any (OK 61x64x12: 0.40 -> 0.19 ms with
// 2 in place of 16).
constexpr int CLUSTER_CHUNK = 16;

// 16 blocks a SM (32 registers): the engine launches 64 warps a SM
__global__ void __launch_bounds__(CLUSTER_WARPS * 32, 16) k_search_cluster(DevJob J, DevPlan P, double *scratch_key,
                                                                      int *scratch_idx, int n_warps_total) {
    __shared__ SortFrame s_stack[CLUSTER_WARPS][SORT_STACK];
    // the partitions' positions by rank, then the tail's keys
    __shared__ double s_buf[CLUSTER_WARPS][SORT_BUF];
    static_assert(SORT_BUF * sizeof(double) >= 128 * sizeof(int), "room for both position lists");
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (gw >= n_warps_total) return;
    const int cap = P.max_candidates;
    double *keys = scratch_key + (long long)gw * cap;
    int *idxs = scratch_idx + (long long)gw * cap;
    const double thr = P.c0 / 100;
    const unsigned below = (1u << lane) - 1;
    // warps take a few consecutive nodes at a time from a counter:
    // clusterizer-path nodes sit in sparse regions, so a fixed share would
    // leave some warps most of them
    const int take = (int)min((long long)CLUSTER_CHUNK, max(1LL, (long long)J.size / (2 * n_warps_total)));
    while (true) {
        int chunk = 0;
        if (lane == 0) chunk = atomicAdd(J.node_next, take);
        chunk = __shfl_sync(FULL_MASK, chunk, 0);
        if (chunk_first(chunk, J.size) >= J.size) break;
        const int chunk_end = (int)min((long long)chunk + take, (long long)J.size);
        for (int node = chunk; node < chunk_end; ++node) {
            if (!node_needs_kriging(J, node)) continue;
            int x, y, z;
            node_xyz(J, node, x, y, z);
            if (!node_clean(P, x, y, z)) continue;
            const int cx = (int)(x / P.crx), cy = (int)(y / P.cry), cz = (int)(z / P.crz);
            int n = 0;
            for (int k = cz - 1; k <= cz + 1; ++k)
                for (int j = cy - 1; j <= cy + 1; ++j) {
                    if (j < 0 || k < 0 || j > P.my || k > P.mz) continue;
                    // the boxes of one row follow one another in the buckets
                    const int i0 = max(cx - 1, 0), i1 = min(cx + 1, P.mx);
                    const long long bi = ((long long)k * P.my + j) * P.mx;
                    const int s0 = P.bucket_start[bi + i0], s1 = P.bucket_start[bi + i1 + 1];
                    int next = s0 + lane < s1 ? __ldg(P.bucket_nodes + s0 + lane) : -1;
                    for (int base = s0; base < s1; base += 32) {
                        const int cand = next;
                        next = base + 32 + lane < s1 ? __ldg(P.bucket_nodes + base + 32 + lane) : -1;
                        bool keep = false;
                        double key = 0;
                        if (cand >= 0) {
                            int dx, dy, dz;
                            node_xyz(J, cand, dx, dy, dz);
                            dx -= x;
                            dy -= y;
                            dz -= z;
                            if (!(reach2(P, (float)dx, (float)dy, (float)dz) > P.reach_limit)) {
                                key = cov_at(P, dx, dy, dz, J.err);
                                keep = key > thr;
                            }
                        }
                        const uint32_t bal = __ballot_sync(FULL_MASK, keep);
                        const int pos = n + __popc(bal & below);
                        if (keep) {
                            if (pos < cap) {
                                keys[pos] = key;
                                idxs[pos] = cand;
                            } else {
                                atomicOr(J.err, DERR_CAND_CAPACITY);
                            }
                        }
                        n += __popc(bal);
                    }
                }
            if (n > cap) n = cap;
            __syncwarp();
            {
                // only the first max_neighbours positions of the reference's sort are used
                SortArr a{keys, idxs};
                int *lbuf = reinterpret_cast<int *>(s_buf[wib]);
                if (!warp_reference_parts(a, n, P.nmax, lane, s_stack[wib], lbuf, lbuf + 64) && lane == 0)
                    atomicOr(J.err, DERR_SORT_STACK);
                warp_sort_tail(a, n, P.nmax, s_buf[wib], J.nb + (long long)node * P.nmax, lane);
            }
            const int cnt = n < P.nmax ? n : P.nmax;
            if (lane == 0) J.nbcount[node] = cnt;
            __syncwarp();
        }
    }
}

// most_probable_category (cdf_utils.cpp:9-24): first maximum wins.
__global__ void k_ik_argmax(DevJob J) {
    long long node = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (node >= J.size) return;
    const float *p = J.probs + node * J.K;
    double best = p[0];
    int bi = 0;
    for (int k = 1; k < J.K; ++k)
        if ((double)p[k] > best) {
            best = p[k];
            bi = k;
        }
    J.out_codes[node] = (uint8_t)bi;
    J.out_mask[node] = 1;
}

// ---------------------------------------------------------------------------
static int sm_count() {
    static const int n = [] {
        int dev = 0, sms = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        return sms > 0 ? sms : 148;
    }();
    return n;
}

void launch_build_bits(const DevJob &J, const DevPlan &P, uint32_t *bits, cudaStream_t s) {
    long long n = (long long)J.ny * J.nz * P.wpr;
    k_build_bits<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(J, P, bits);
}

void launch_search_template(const DevJob &J, const DevPlan &P, cudaStream_t s) {
    const long long segs = (long long)P.nseg * J.ny * J.nz;
    long long blocks = (segs + 7) / 8;
    const long long cap = (long long)sm_count() * 8;  // 8 blocks of 8 warps per SM
    if (blocks > cap) blocks = cap;
    k_search_template<<<(unsigned)std::max<long long>(1, blocks), 256, 0, s>>>(J, P);
}

void launch_search_cluster(const DevJob &J, const DevPlan &P, double *sk, int *si, int n_warps, cudaStream_t s) {
    const int threads = CLUSTER_WARPS * 32;
    k_search_cluster<<<(unsigned)((n_warps * 32 + threads - 1) / threads), threads, 0, s>>>(J, P, sk, si, n_warps);
}

void launch_solve(const DevJob &J, const DevPlan &P, cudaStream_t s, int blocks_per_sm) {
    if (J.size <= 0) return;
    if (P.nmax <= 32) launch_solve32(J, P, s, blocks_per_sm);
    else launch_solve64(J, P, s, blocks_per_sm);
}

// ---------------------------------------------------------------------------
// Speculative sequential simulation: path ranks, commits and admissions (the
// rounds' kriging is launch_sgs_try32 / launch_sgs_try64 in the solve files).

__global__ void k_sgs_rank_init(DevJob J, int *rank_of) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i < J.size) rank_of[i] = J.mask[i] ? -1 : INT_MAX;
}

__global__ void k_sgs_rank_path(const int *nodes, int *rank_of, long long nsim) {
    const long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (r < nsim) rank_of[nodes[r]] = (int)r;
}

__device__ __forceinline__ void sgs_bit(const DevJob &J, const DevPlan &P, int node, long long &w, uint32_t &bit) {
    int x, y, z;
    node_xyz(J, node, x, y, z);
    const int px = x + P.px;
    w = ((long long)z * J.ny + y) * P.wpr + (px >> 5);
    bit = 1u << (px & 31);
}

// Place of this thread's entry in a list that the block appends to: one
// update of the list's counter a block (a warp each, 8 192 updates of one
// address a pass over the window, took longer than the pass itself).  Every
// thread of the block calls it, `want` or not.
__device__ __forceinline__ int block_append(bool want, int *counter, int (&warp_at)[8]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned m = __ballot_sync(FULL_MASK, want);
    if (lane == 0) warp_at[warp] = __popc(m);
    __syncthreads();
    if (threadIdx.x == 0) {
        int total = 0;
        for (int w = 0; w < 8; ++w) {
            const int c = warp_at[w];
            warp_at[w] = total;
            total += c;
        }
        const int at = total ? atomicAdd(counter, total) : 0;
        for (int w = 0; w < 8; ++w) warp_at[w] += at;
    }
    __syncthreads();
    const int at = warp_at[warp] + __popc(m & ((1u << lane) - 1u));
    __syncthreads();
    return at;
}

// The round's try list: the pending nodes of window buffer `cur` without a
// blocker or whose blocker has committed; the others stay pending untried.
__global__ void __launch_bounds__(256) k_sgs_list(SgsState G, int cur) {
    __shared__ int warp_at[8];
    SgsCtl *ctl = G.ctl;
    const int count = ctl->count[cur];
    const int *win = cur ? G.win1 : G.win0;
    const int stride = gridDim.x * 256;
    for (int base = blockIdx.x * 256; base < count; base += stride) {
        const int i = base + (int)threadIdx.x;
        bool tr = false;
        if (i < count) {
            const int b = G.blocker[win[i]];
            tr = b < 0 || G.done[b];
            if (!tr) G.ok[i] = 0;
        }
        const int at = block_append(tr, &ctl->ntry, warp_at);
        if (tr) G.trylist[at] = i;
    }
}

// Commits the nodes of window buffer `cur` that the round kept (informed bit
// set, pending bit cleared, done) and moves the others to the other buffer.
// The last block to finish (a ticket counter, no waiting) tops the window up
// to its size and records the admission that k_sgs_admit carries out.
__global__ void __launch_bounds__(256) k_sgs_commit(DevJob J, DevPlan P, SgsState G, int cur) {
    __shared__ int warp_at[8];
    SgsCtl *ctl = G.ctl;
    const int count = *(volatile int *)&ctl->count[cur];
    const int *win = cur ? G.win1 : G.win0;
    int *nxt = cur ? G.win0 : G.win1;
    const int stride = gridDim.x * 256;
    for (int base = blockIdx.x * 256; base < count; base += stride) {
        const int i = base + (int)threadIdx.x;
        int rank = -1;
        bool keep = false;
        if (i < count) {
            rank = win[i];
            if (G.ok[i]) {
                long long w;
                uint32_t bit;
                sgs_bit(J, P, G.nodes[rank], w, bit);
                atomicOr(J.sim_bits + w, bit);
                atomicAnd(G.pend + w, ~bit);
                G.done[rank] = 1;
            } else {
                keep = true;
            }
        }
        const int at = block_append(keep, &ctl->count[cur ^ 1], warp_at);
        if (keep) nxt[at] = rank;
    }
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(&ctl->blocks_done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last || threadIdx.x != 0) return;
    __threadfence();
    const int kept = atomicAdd(&ctl->count[cur ^ 1], 0);
    long long add = (long long)ctl->window - kept;
    if (add < 0) add = 0;
    if (add > ctl->total - ctl->next) add = ctl->total - ctl->next;
    ctl->admit_base = kept;
    ctl->admit = add;
    ctl->next += add;
    ctl->count[cur ^ 1] = kept + (int)add;
    ctl->count[cur] = 0;
    if (count > 0) {
        ctl->rounds += 1;
        ctl->commits += count - kept;
    }
    ctl->tries += ctl->ntry;
    ctl->ntry = 0;
    ctl->nsolve = 0;
    ctl->blocks_done = 0;
    ctl->cursor = 0;
    ctl->solve_cursor = 0;
}

// Appends the admitted path ranks to window buffer `buf` and marks them
// pending.
__global__ void __launch_bounds__(256) k_sgs_admit(DevJob J, DevPlan P, SgsState G, int buf) {
    const SgsCtl *ctl = G.ctl;
    const long long add = ctl->admit, base = ctl->admit_base, first = ctl->next - add;
    int *win = buf ? G.win1 : G.win0;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < add;
         k += (long long)gridDim.x * blockDim.x) {
        const int rank = (int)(first + k);
        win[base + k] = rank;
        long long w;
        uint32_t bit;
        sgs_bit(J, P, G.nodes[rank], w, bit);
        atomicOr(G.pend + w, bit);
    }
}

void launch_sgs_ranks(const DevJob &J, const SgsState &G, long long nsim, cudaStream_t s) {
    int *rank_of = const_cast<int *>(G.rank_of);
    k_sgs_rank_init<<<(unsigned)((J.size + 255) / 256), 256, 0, s>>>(J, rank_of);
    if (nsim > 0) k_sgs_rank_path<<<(unsigned)((nsim + 255) / 256), 256, 0, s>>>(G.nodes, rank_of, nsim);
}

static void sgs_commit_admit(const DevJob &J, const DevPlan &P, const SgsState &G, int cur, cudaStream_t s) {
    const unsigned blocks = (unsigned)sm_count() * 4;
    k_sgs_commit<<<blocks, 256, 0, s>>>(J, P, G, cur);
    k_sgs_admit<<<blocks, 256, 0, s>>>(J, P, G, cur ^ 1);
}

void launch_sgs_admit(const DevJob &J, const DevPlan &P, const SgsState &G, int cur, cudaStream_t s) {
    sgs_commit_admit(J, P, G, cur, s);
}

static void sgs_list(const SgsState &G, int cur, cudaStream_t s) {
    k_sgs_list<<<(unsigned)sm_count() * 4, 256, 0, s>>>(G, cur);
}

void launch_sis_round(const DevJob &J, const DevPlan &P0, const DevPlan *plans, int family, const SisGroups &groups,
                      const SgsState &G, int cur, cudaStream_t s) {
    sgs_list(G, cur, s);
    if (groups.n > 0) launch_sis_groups(J, groups, G, cur, s);
    else if (family == 0) launch_sis_try32(J, plans, G, cur, s);
    else launch_sis_try64(J, plans, G, cur, s);
    sgs_commit_admit(J, P0, G, cur, s);
}

void launch_sgs_round(const DevJob &J, const DevPlan &P, const SgsState &G, int cur, cudaStream_t s) {
    sgs_list(G, cur, s);
    if (P.nmax <= 32) launch_sgs_try32(J, P, G, cur, s);
    else launch_sgs_try64(J, P, G, cur, s);
    sgs_commit_admit(J, P, G, cur, s);
}

long long persistent_grid(const void *fn, int threads, size_t smem, int blocks_per_sm, long long units) {
    // occupancy of each kernel is looked up once
    static std::mutex mu;
    static std::map<const void *, int> occ;
    int per_sm;
    {
        std::lock_guard<std::mutex> lock(mu);
        auto it = occ.find(fn);
        if (it == occ.end()) {
            cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            int v = 0;
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, fn, threads, smem);
            it = occ.emplace(fn, v < 1 ? 1 : v).first;
        }
        per_sm = it->second;
    }
    if (blocks_per_sm > 0 && blocks_per_sm < per_sm) per_sm = blocks_per_sm;
    const long long cap = (long long)per_sm * sm_count();
    return std::max<long long>(1, std::min(units, cap));
}

namespace {
std::mutex g_tuning_mu;
LaunchTuning g_tuning[2][2];
}  // namespace

LaunchTuning tuning_get(int family, int precision) {
    std::lock_guard<std::mutex> lock(g_tuning_mu);
    return g_tuning[family & 1][precision & 1];
}

void tuning_set(int family, int precision, const LaunchTuning &t) {
    std::lock_guard<std::mutex> lock(g_tuning_mu);
    g_tuning[family & 1][precision & 1] = t;
}

void launch_ik_argmax(const DevJob &J, cudaStream_t s) {
    k_ik_argmax<<<(unsigned)((J.size + 255) / 256), 256, 0, s>>>(J);
}

}  // namespace hpgl_b200
