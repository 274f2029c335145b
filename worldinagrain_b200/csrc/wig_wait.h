// wig_wait.h — the word a grid barrier's CTAs count their arrivals in, and
// give up by.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define WIG_WAIT_FN __host__ __device__ constexpr
#else
#define WIG_WAIT_FN constexpr
#endif

namespace wig {

// An arrival adds 1 to the word; the k-th barrier of a grid of n CTAs is
// passed at k n arrivals (at most 148 x 64 iterations x about 30 barriers: far
// below the mark).  A CTA whose wait runs out ORs the mark in: any number of
// CTAs may, and the word then reads as given up for good, whatever arrivals
// are still added to it.  (Added as a number, the mark of a fourth CTA wrapped
// the word round and took the others' away, so that waits after it ran to
// their limit again, or passed.)
constexpr uint32_t BARRIER_GAVE_UP = 1u << 31;

WIG_WAIT_FN bool barrierGaveUp(uint32_t word) { return (word & BARRIER_GAVE_UP) != 0u; }
// Whether a wait for `target` arrivals is over, one way or the other.
WIG_WAIT_FN bool barrierOver(uint32_t word, uint32_t target) { return barrierGaveUp(word) || word >= target; }

}  // namespace wig
