// wig_fast.cuh — the fast form of the pressure solve: the same arithmetic as
// the reference's CG / V-cycle passes (fluid.wgsl:2047-2893), over
// structure-of-arrays scratch with the stencil's coefficients worked out once
// a step, its iterations looped on the device by a CUDA-graph WHILE node, one
// launch a pass for all the worlds of a batch.
#pragma once
#include "wig_passes.cuh"

namespace wig {

// The one-CTA coarse kernel (and CTA 0 of a world's solve in one launch)
// holds levels of at most this many cells.
constexpr uint32_t COARSE_CTA_CELLS = 4096;
// A single world's coarse levels from a level of up to this many cells run
// on a thread-block cluster (k_fCoarseCluster).
constexpr uint32_t COARSE_CLUSTER_CELLS = 16384;

// A world's first level of at most `cells` cells (its coarsest when none
// above it is): where the coarse kernel takes over.
inline uint32_t coarse_level(const Dev& D, uint32_t cells) {
    for (uint32_t l = 1; l <= D.levels; l++)
        if ((size_t)D.level_w[l] * D.level_h[l] <= cells) return l;
    return D.levels;
}
// The most dynamic shared memory a CTA of these kernels takes.
constexpr size_t SOLVE_SMEM_MOST = 220u * 1024u;

// How a single world's solve in one launch is shaped: the CTAs of a
// cooperative grid; the CTAs of one cluster (0: the world has too many
// blocks for one); the first level that fits one CTA.
struct SolveShape {
    uint32_t grid, cluster, lc;
};
constexpr uint32_t SOLVE_CLUSTER = 16;
// A single world of up to CLUSTER_BLOCKS blocks solves in one launch, on a
// cluster, whose barrier is the cheapest but whose 16 multiprocessors are few
// (a step of a pond of 75x52 200 us against 218 as the loop's launches, of the
// dam at 192x192 673 against 724, of two liquids at 224x224 928 against 890).
// One of more than GRID_BLOCKS does so on a grid of all the multiprocessors,
// stepped on the legacy stream: 5-9% faster at 640x640 to 1024x1024 (the disks
// at 1024x1024 4617 us a step against 5034 as the loop's launches; at 512x512
// 1595 against 1554, the dam at 520x520 814 against 791, the 2048x2048 column
// 11330 against 11220).  Nothing else runs beside such a solve, so a world
// stepped on a stream of its own, as a host gives one that it means to run
// beside other work, keeps the loop's launches: two dams at 520x520 at once
// take 489 us a step each so and 756 with grids, four 323 and 724, four of the
// disks at 1024x1024 3170 and 4660.
constexpr uint32_t CLUSTER_BLOCKS = 640, GRID_BLOCKS = 4096;
// A grid's CTAs: a tile of the fine level for every other warp, at most a
// CTA a multiprocessor (a tile a warp is 1% slower at 256x256, 4 or 8 tiles
// a CTA the same).
constexpr uint32_t GRID_TILES = 16;

// A profiler's hook around each launch: fn(ctx, slot, 0) before, (ctx, slot, 1) after.
struct Marker {
    void (*fn)(void* ctx, int slot, int phase);
    void* ctx;
};

// While an iteration is captured into the loop's body graph: a stream for
// the bodies of the conditional nodes inside it (the mixed form's
// true-residual check and fix run in IF nodes, so the iterations that need
// neither launch neither), and the first CUDA error met.
struct NestCapture {
    cudaStream_t s;
    cudaError_t err;
};

// Launchers over a batch (stream-ordered; all capturable).  `one`: the
// batch's only world (host copy), passed to the kernels as a parameter; null
// for a batch of several.  fast_cycle returns the launches every iteration
// makes; `nest`: the capture's stream for conditional bodies (null when
// launched eagerly: the check and the fix are then launched every
// iteration and return at once when not needed).
void fast_setup(const Batch& Bt, const BatchShape& S, const World* one, cudaStream_t s, const Marker* m);
uint32_t fast_cycle(const Batch& Bt, const BatchShape& S, const World* one, cudaStream_t s, const Marker* m,
                    NestCapture* nest = nullptr);
// cgFinish.
void fast_finish(const Batch& Bt, const BatchShape& S, const World* one, cudaStream_t s, const Marker* m);
// Level 0's arrays of one world zeroed (after its buffers are written by the host).
void fast_zero_level0(const World& Wd, cudaStream_t s);
// The same for the blocks not worked on, of every world of the step whose
// scratch a pool lends (after compact).
void fast_zero_idle(const Batch& Bt, const BatchShape& S, cudaStream_t s);
// Shared memory of the coarse kernel for a world, and the kernel's limit set.
size_t fast_coarse_smem(const Dev& D, uint32_t lc);
// Shared memory a CTA of the cluster coarse kernel takes for a single world
// from level lc; 0 when that kernel does not apply (level lc fits the one-CTA
// kernel, or the world's coarsest level does not fit one CTA of the cluster).
size_t fast_cluster_smem(const Dev& D, uint32_t lc);
cudaError_t fast_prepare_attributes();
// A single world's solve: all its iterations in one launch, on one cluster
// or (`grid`, or no cluster fits it) a cooperative grid.
cudaError_t fast_solve_shape(const Dev& D, SolveShape* out);
cudaError_t fast_solve(const Batch& Bt, const World& W0, const SolveShape& h, bool grid, cudaStream_t s, const Marker* m);

}  // namespace wig
