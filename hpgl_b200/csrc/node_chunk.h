// Chunks of nodes handed out by a counter, compiled for host and device.  Each
// warp of a launch takes one chunk too many, so near 2^31 nodes the counter runs
// past the largest int and comes back negative, and the last chunk's end lies
// beyond it.
#pragma once

#ifdef __CUDACC__
#define HPGL_CHUNK_HD __host__ __device__ __forceinline__
#else
#define HPGL_CHUNK_HD inline
#endif

namespace hpgl_b200 {

// The chunk's first node, or `size` when the nodes have been handed out.
HPGL_CHUNK_HD long long chunk_first(int counter, long long size) {
    return counter >= 0 && counter < size ? counter : size;
}

// Whether the chunk from `first` (one of the nodes) has an l-th node.
HPGL_CHUNK_HD bool chunk_has(int first, int l, int chunk, long long size) { return l < chunk && l < size - first; }

}  // namespace hpgl_b200
