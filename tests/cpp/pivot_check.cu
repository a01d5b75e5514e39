// Compares sqrt_rcp (hpgl_b200/csrc/tile_solve.cuh: root and reciprocal root
// together) and recip (cok_tile.cuh: a reciprocal of either sign) with CUDA's IEEE operations __dsqrt_rn and __drcp_rn on the GPU:
// operands of kriging pivots' magnitudes, over sqrt_rcp's whole range, next to
// squares of short numbers (roots near rounding boundaries), and next to the
// squares of the numbers just below powers of two (divisors with a
// significand of ones).  Prints the mismatches and exits non-zero on any.
#include <cstdio>
#include <cstdlib>
#include "../../hpgl_b200/csrc/cok_tile.cuh"
#include "../../hpgl_b200/csrc/tile_solve.cuh"

__device__ unsigned long long g_bad;

__device__ __forceinline__ unsigned long long mix(unsigned long long x) {
    x ^= x >> 33; x *= 0xff51afd7ed558ccdULL; x ^= x >> 33; x *= 0xc4ceb9fe1a85ec53ULL; x ^= x >> 33;
    return x;
}
__device__ __forceinline__ double with_exponent(unsigned long long m, int e) {
    return __longlong_as_double((long long)((m & 0x000FFFFFFFFFFFFFULL) | ((unsigned long long)(1023 + e) << 52)));
}

__global__ void check(unsigned long long n, unsigned long long seed, int what) {
    unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
    const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
    unsigned long long bad = 0;
    for (; i < n; i += stride) {
        const unsigned long long u = mix(i * 2 + seed), v = mix(i * 2 + 1 + seed);
        double a;
        if (what == 0) {
            a = with_exponent(u, -(int)(v % 56)) * 2.0;
        } else if (what == 1) {
            a = with_exponent(u, -760 + (int)(v % 1520));
        } else if (what == 2) {
            const double s = with_exponent((u >> 26) << 26, -20 + (int)(v % 40));  // 26 bits: an exact square
            a = __longlong_as_double(__double_as_longlong(s * s) + (long long)(v >> 40) % 9 - 4);
        } else {
            const double s = with_exponent(~0ULL - (u % 4), -200 + (int)(v % 400));
            a = __longlong_as_double(__double_as_longlong(s * s) + (long long)(v >> 40) % 9 - 4);
        }
        double root, rcp;
        hpgl_b200::sqrt_rcp(a, root, rcp);
        const double r = __dsqrt_rn(a), q = __drcp_rn(r);
        // the reciprocal of the root and of the operand, with a random sign
        const double b = (v & 1) ? -root : (v & 2) ? -a : a;
        double p;
        if (!hpgl_b200::recip(b, p) || __double_as_longlong(p) != __double_as_longlong(__drcp_rn(b))) ++bad;
        if (__double_as_longlong(r) != __double_as_longlong(root) || __double_as_longlong(q) != __double_as_longlong(rcp)) ++bad;
    }
    if (bad) atomicAdd(&g_bad, bad);
}

int main(int argc, char **argv) {
    const unsigned long long n = argc > 1 ? strtoull(argv[1], 0, 10) : 100000000ULL;
    const char *names[] = {"pivots", "whole range", "near squares", "roots of ones"};
    unsigned long long total = 0;
    for (int what = 0; what < 4; ++what) {
        unsigned long long bad = 0;
        cudaMemcpyToSymbol(g_bad, &bad, sizeof(bad));
        check<<<1184, 256>>>(n, 98765 + what, what);
        if (cudaDeviceSynchronize() != cudaSuccess) { printf("cuda error\n"); return 2; }
        cudaMemcpyFromSymbol(&bad, g_bad, sizeof(bad));
        printf("%s: mismatches %llu of %llu\n", names[what], bad, n);
        total += bad;
    }
    return total ? 1 : 0;
}
