// Device helpers shared by the kernel files.
#pragma once
#include <cstdint>

#include "kernels.cuh"
#include "node_chunk.h"

namespace hpgl_b200 {

#define FULL_MASK 0xffffffffu

// kinds with a continuous property: OK, SK, LVM and the two cokriging kinds
__device__ __forceinline__ bool is_cont(int kind) { return kind <= 2 || kind == 5 || kind == 6; }

// Covariance of offset v (grid steps) from the plan's table.  Truncated kinds
// read 0 beyond the search radii (precalculated_covariance.h:60-75,
// covariance_field.h:144-153); the table box covers every offset the search
// can produce, anything else is a broken invariant.
// For truncated kinds T = min(radii, B) and every |v| <= n-1 <= B, so the
// table covers all in-radius offsets; for ordinary kriging T = B covers
// every offset the search produces (an offset beyond it raises an error bit).
__device__ __forceinline__ bool cov_in_range(const DevPlan &P, int vx, int vy, int vz) {
    return (unsigned)(vx + P.Tx) <= (unsigned)(2 * P.Tx) && (unsigned)(vy + P.Ty) <= (unsigned)(2 * P.Ty) &&
           (unsigned)(vz + P.Tz) <= (unsigned)(2 * P.Tz);
}

// lin = vz*syx + vy*sx + vx, the table offset of v; C(v) = C(-v) bit for bit, and
// the table holds the offsets of lin >= 0.
__device__ __forceinline__ double cov_lin(const DevPlan &P, int vx, int vy, int vz, int lin, int *err) {
    if (!cov_in_range(P, vx, vy, vz)) {
        if (!P.truncated) atomicOr(err, DERR_TABLE_RANGE);
        return 0.0;
    }
    return __ldg(P.table + abs(lin));
}

__device__ __forceinline__ double cov_at(const DevPlan &P, int vx, int vy, int vz, int *err) {
    return cov_lin(P, vx, vy, vz, vz * P.syx + vy * P.sx + vx, err);
}

// Node coordinates, sugarbox_grid.cpp:70-74 (x = idx % nx, y = idx % (nx ny) / nx,
// z = idx / (nx ny)), with the two divisions by multiply-high.
__device__ __forceinline__ void node_xyz(const DevJob &J, int idx, int &x, int &y, int &z) {
    const unsigned r = J.div_nx.div((unsigned)idx);
    const unsigned q = J.div_ny.div(r);
    x = idx - (int)r * J.nx;
    y = (int)r - (int)q * J.ny;
    z = (int)q;
}

// A node takes the template walk when any of its 27 neighbouring clusterizer
// boxes overflowed (sugarbox_indexed_neighbour_lookup.h:68-71).
__device__ __forceinline__ bool node_clean(const DevPlan &P, int x, int y, int z) {
    int cx = (int)(x / P.crx), cy = (int)(y / P.cry), cz = (int)(z / P.crz);
    return P.bucket_clean[((long long)cz * P.my + cy) * P.mx + cx] != 0;
}

__device__ __forceinline__ bool node_needs_kriging(const DevJob &J, int node) {
    return is_cont(J.kind) ? J.mask[node] == 0 : true;
}

// Correctly rounded quotient a / b from y = RN(1/b): q = RN(a*y) is within
// one ulp of a/b, r = a - b*q is exact in one fused multiply-add, and
// RN(q + r*y) is the correctly rounded quotient (Markstein's theorem, IBM J.
// Res. Dev. 34(1), 1990, for round-to-nearest binary arithmetic away from
// overflow and the subnormal range).  Bit-identical to __ddiv_rn on the
// kriging systems' magnitudes; tests/test_division.py checks it against
// __ddiv_rn on the GPU.
__device__ __forceinline__ double div_by_rcp(double a, double b, double y) {
    const double q = __dmul_rn(a, y);
    const double r = __fma_rn(-q, b, a);
    return __fma_rn(r, y, q);
}

// The first loads of a node, issued one node ahead by the persistent loops
// (the neighbour count, the lane's neighbour cells -- rows lane and lane + 32
// -- and the informed flag start a chain of dependent loads; issuing them
// while the previous system is solved hides that latency).  Plain loads: the
// fused kernels read lists their own warp has just written.
struct NodeFetch {
    int node;  // -1: past the end
    int n;
    int cell, cell2;
    bool informed;
};

__device__ __forceinline__ NodeFetch fetch_node(const DevJob &J, const DevPlan &P, int node, int lane) {
    NodeFetch f;
    f.node = node;
    f.n = 0;
    f.cell = 0;
    f.cell2 = 0;
    f.informed = false;
    if (node >= 0) {
        f.n = J.nbcount[node];
        const int *lst = J.nb + (long long)node * P.nmax;
        if (lane < P.nmax) f.cell = lst[lane];
        if (lane + 32 < P.nmax) f.cell2 = lst[lane + 32];
        f.informed = is_cont(J.kind) && __ldg(J.mask + node) != 0;
    }
    return f;
}

// Nodes a solve warp takes from the per-job counter at a time: up to `cap`,
// fewer on small jobs so that every warp of the grid still gets about 8
// chunks (the size depends only on the job and the launch).
__device__ __forceinline__ int chunk_nodes(const DevJob &J, int cap, int warps_per_block) {
    const long long c = J.size / ((long long)gridDim.x * warps_per_block * 8);
    return (int)(c < 1 ? 1 : (c > cap ? cap : c));
}

}  // namespace hpgl_b200
