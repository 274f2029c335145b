// wig_sums.cuh — sums over a world's blocks in the reference's fixed order: a
// block's tree of 64 by a warp, the block partials' columns and tree by a CTA.
#pragma once
#include "wig_device.cuh"

namespace wig {
namespace {

// A tile's tree of 64 (sumBlock, fluid.wgsl:2628-2641) from a lane's two
// values; the sum in lane 0.
template <class T>
__device__ __forceinline__ T warpTree(T lo, T hi) {
    T v = lo + hi;
#pragma unroll
    for (int h = 16; h > 0; h >>= 1) v = v + __shfl_down_sync(0xffffffffu, v, h);
    return v;
}

// The tree of 256 of NC components' column sums, a component's at s + 256 c,
// written by the CTA's threads; the sums in s[256 c], for every thread.
template <class T, int NC>
__device__ __forceinline__ void treeColumns(T* s) {
    const uint32_t li = threadIdx.x & 255u, c = threadIdx.x >> 8;
    T* own = s + 256u * c + li;
    __syncthreads();
#pragma unroll
    for (uint32_t h = 128u; h > 32u; h >>= 1) {
        if (c < NC && li < h) *own = *own + own[h];
        __syncthreads();
    }
    if (c < NC && li < 32u) {
        T v = *own + own[32];
#pragma unroll
        for (int h = 16; h > 0; h >>= 1) v = v + __shfl_down_sync(0xffffffffu, v, h);
        if (li == 0u) *own = v;
    }
    __syncthreads();
}

// sumBlocks (fluid.wgsl:2645-2661) of the first NC components of a world's
// B block partials by a CTA of NT threads: column li (of 256) adds blocks
// li, li + 256, ... in that order, 16 rows' loads in flight a thread, the
// CTA's groups of 256 threads sharing the components and, NT / 256 / NC a
// component, taking 16 rows each of a column in turn and passing its sum on,
// so the order of the adds stays.  A block not worked on has partials of
// +0, and a sum that starts from +0 is never -0, so adding them changes no
// bit: its state is not read.  The sums in s[256 c], for every thread.
template <class T, int NC, int NT>
__device__ __noinline__ void sumColumns(uint32_t B, const T* part, T* s) {
    constexpr uint32_t ROWS = 16u, SPAN = 256u * ROWS, TURNS = NT / 256 / NC;
    const uint32_t li = threadIdx.x & 255u, group = threadIdx.x >> 8;
    const uint32_t c = group / TURNS, turn = group % TURNS;
    T* own = s + 256u * c + li;
    const T* at = part + (size_t)B * c;
    T acc = T(0);
    for (uint32_t r0 = 0; r0 < B; r0 += TURNS * SPAN) {
        T v[ROWS];
        const uint32_t k0 = r0 + turn * SPAN + li;
#pragma unroll
        for (uint32_t u = 0; u < ROWS; u++) v[u] = k0 + 256u * u < B ? __ldcg(at + k0 + 256u * u) : T(0);
#pragma unroll
        for (uint32_t t = 0; t < TURNS; t++) {
            if (t > 0u && r0 + t * SPAN >= B) break;  // (uniform: no more rows)
            if (t > 0u) __syncthreads();
            if (turn == t) {
                if (t > 0u || (TURNS > 1u && r0 > 0u)) acc = *own;
#pragma unroll
                for (uint32_t u = 0; u < ROWS; u++) acc = acc + v[u];
                if (TURNS > 1u) *own = acc;
            }
        }
        if (TURNS > 1u) __syncthreads();
    }
    if (TURNS == 1u) *own = acc;
}
}  // namespace
}  // namespace wig
