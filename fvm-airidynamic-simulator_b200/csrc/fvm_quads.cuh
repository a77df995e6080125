// fvm_quads.cuh -- access to a whole state four cells at a time, and the
// last-block pattern of the reductions over it.
#pragma once
#include <algorithm>

#include "fvm_internal.cuh"

namespace fvm {

// Whole-field passes work on groups of four neighbouring cells of a row: a
// state's rows start 128-byte aligned (pitch a multiple of 32 floats), so a
// group is one 16-byte load per plane and one 4-byte load of mask bytes, and
// every load of a group is issued before anything depends on one.  The last
// group of a row may reach into the row's padding; its cells beyond nx are
// loaded and ignored.
struct Quad {
    int j, i, n;   // row, first column, cells inside the grid (1..4)
    size_t c, d;   // pitched and dense index of the first cell
};
__host__ __device__ __forceinline__ unsigned quads_per_row(const GridDesc &g) { return (unsigned)(g.nx + 3) / 4u; }
// groups of a grid (fewer than 2^31 cells, so fewer than 2^31 groups)
__host__ __device__ __forceinline__ unsigned quads(const GridDesc &g) { return quads_per_row(g) * (unsigned)g.ny; }
__device__ __forceinline__ Quad quad_at(const GridDesc &g, unsigned e) {
    const unsigned per = quads_per_row(g);
    Quad q;
    q.j = (int)(e / per);
    q.i = (int)(e % per) * 4;
    q.n = min(4, g.nx - q.i);
    q.c = (size_t)q.j * g.pitch + q.i;
    q.d = (size_t)q.j * g.nx + q.i;
    return q;
}
__device__ __forceinline__ float4 load4(const float *plane, const Quad &q) {
    return __ldg(reinterpret_cast<const float4 *>(plane + q.c));
}
__device__ __forceinline__ float lane4(const float4 &v, int k) { return k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w; }

// True in every thread of the one block that arrives last; what the other
// blocks wrote before is then visible to it.  The counter is zero again after.
__device__ __forceinline__ bool last_block(unsigned *counter) {
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(counter, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return false;
    if (threadIdx.x == 0) *counter = 0u;
    __threadfence();
    return true;
}

// blocks of 256 threads over a grid's groups of four cells, at most `cap`
inline unsigned quad_blocks(const GridDesc &g, unsigned cap) {
    return std::max(1u, std::min(cap, (quads(g) + 255u) / 256u));
}
// one group per thread
inline unsigned quad_blocks(const GridDesc &g) { return (quads(g) + 255u) / 256u; }
}  // namespace fvm
