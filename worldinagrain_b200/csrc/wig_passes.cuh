// wig_passes.cuh — launchers of the liquid step's pass kernels.
#pragma once
#include "wig_device.cuh"

namespace wig {

// Host-side shape of a batch: the most items each work list can hold (grid
// sizes of the kernels over it).
struct BatchShape {
    uint32_t max_items[L_COUNT];
    uint32_t worlds;
    uint32_t levels;       // deepest coarse level of any world
    uint32_t lc_max;       // deepest level any world restricts by itself
    size_t coarse_smem;    // the coarse kernel's shared memory for the largest world (a CTA's, on a cluster)
    uint32_t cluster;      // a single world's coarse levels on a thread-block cluster
    // launch shapes (wig_launch_knob): none changes a result
    uint32_t coarse_cells;  // the coarse kernel from a world's first level of at most this many cells
    uint32_t level_per_sm, cg_per_sm, relax_per_sm;
};

// CTAs for a kernel over list `list` with `per_sm` CTAs a multiprocessor.
unsigned list_grid(const BatchShape& S, uint32_t list, unsigned per_sm);

// A solve pass's `cycle` in a step's loop: the iteration the world's
// StepState says (a pass of that iteration, not converged before it).
constexpr uint32_t CYCLE_LOOP = 0xffffffffu;

// One reference pass (enum wig_pass) at Level (level, cycle), on stream s:
// over the batch's work lists, or (the plain form's solve passes) over
// world 0, whose descriptor D0 is.  `one`: the batch's only world (host
// copy), passed to the kernels as a parameter, so that no CTA starts by
// loading the world's entry (33 launches of a step of a small world each
// spent about 1 us of their 4-5 on it); null for a batch of several.
int launch_pass(const Batch& Bt, const BatchShape& S, const World* one, const Dev& D0, int pass, uint32_t level,
                uint32_t cycle, cudaStream_t s);
// Device-side report of a world: the FLUID_COUNT words, the particle count
// and the solve's residuals, gathered at the end of a step.
struct Report {
    uint32_t count[WIG_FLUID_STATS];
    uint32_t particles;
    uint32_t err;
    uint32_t short_of_tol;  // a tolerance-form solve of a nonzero b stopped above its tolerance
    uint32_t tried;         // particles the step's sync and seeding put into `parts` (past its room: lost)
    double rel;
    double bnorm2;
    double rel_true;
};
// Where a step's reports go: by the world, and by its place in the step's list.
struct ReportTo {
    Report* by_world;
    Report* by_entry;
};
// A step's own forms of some passes, which take in others: retire with the
// reports (a bookkeeping-only step's last pass), clear with retire,
// divergence with cgStart (its block's own labelling), cgJoin across the
// blocks (the same regions and roots as cgStart and cgJoin), advect with
// sortCount, scatter from the blocks' places, rasterClaims with scanFinish,
// unpaint with the reports.  Each took a launch of 2.5-4 us on a small
// world, and on a large one a pass over its words.
void launch_step_pass(const Batch& Bt, const BatchShape& S, const World* one, const ReportTo& to, int pass, cudaStream_t s);
// Whether a single world's compact is two launches.
bool compact_split(const World* one);
// The plain form's ||b||^2 of world 0 after cgResidual (the tolerance form).
void launch_norm(const Dev& D, cudaStream_t s);
// The end of an iteration of the plain form's loop on world 0, after
// cgUpdate: the tolerance form's ||r||/||b||, and the loop's verdict into
// Bt.loop and the WHILE node's condition Bt.cond (0: none).
void launch_cycle_end(const Batch& Bt, const Dev& D, cudaStream_t s);
}  // namespace wig
