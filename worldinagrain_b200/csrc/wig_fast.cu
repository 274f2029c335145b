// wig_fast.cu — the fast form of the liquid's pressure solve (the CG loop
// of encodeFluid, js/sim.js:2551-2591; fluid.wgsl:2047-2893).
//
// Same arithmetic as the reference's passes, operation for operation and in
// the same order (so every value the step leaves is bit-for-bit the plain
// form's), arranged for the GPU:
//   * the stencil's coefficients (fineBeta on the cells, faceBeta on the
//     coarse levels) are worked out once a step and kept, instead of being
//     recomputed with their divisions in every sweep;
//   * the vectors live in structure-of-arrays scratch (a float per cell,
//     row-major), so a warp's loads are contiguous instead of 32-44 bytes
//     apart as in the reference's per-cell records;
//   * the levels of at most 4096 cells, down to the coarsest and back, are
//     one CTA's work in shared memory, one launch instead of ~15;
//   * the CG's block sums finish in the last block to write its partial (a
//     threadfence reduction: the same fixed tree order, one launch fewer);
//   * the iterations are the body of a CUDA-graph WHILE node: a step runs as
//     many as it needs, with no launches for the converged ones.
// The scratch keeps one invariant: level-0 arrays are zero outside the blocks
// worked on (zeroed at allocation, when a world is uploaded, and by retire,
// in whichever form's step, which zeroes the reference's field there too), and
// so are the blocks' partial sums (zeroed by each step's set-up).

#include <algorithm>

#include <cooperative_groups.h>
#include <cuda_bf16.h>

#include "wig_bodies.cuh"
#include "wig_fast.cuh"
#include "wig_sums.cuh"
#include "wig_wait.h"

namespace wig {
namespace {

__device__ __forceinline__ uint32_t vld(const uint32_t* p) { return *(const volatile uint32_t*)p; }

__device__ __forceinline__ I2 lidCell(const W& w, uint32_t wid) {
    I2 b = w.activeBlock(wid);
    return I2{b.x * BLOCK + (int)(threadIdx.x & 7u), b.y * BLOCK + (int)(threadIdx.x >> 3)};
}

// Neighbour d (left, right, up, down: beside, fluid.wgsl:267-269) of cell
// (x, y) on a w x h level, clamped onto the cell itself past the edge (its
// coefficient there is 0).
__device__ __forceinline__ uint32_t nbr(uint32_t i, int x, int y, int w, int h, int d) {
    switch (d) {
    case 0: return x > 0 ? i - 1u : i;
    case 1: return x < w - 1 ? i + 1u : i;
    case 2: return y > 0 ? i - (uint32_t)w : i;
    default: return y < h - 1 ? i + (uint32_t)w : i;
    }
}
__device__ __forceinline__ bool nbrIn(int x, int y, int w, int h, int d) {
    switch (d) {
    case 0: return x > 0;
    case 1: return x < w - 1;
    case 2: return y > 0;
    default: return y < h - 1;
    }
}

// A 256-thread CTA's four trees of 64 (sumBlock's, fluid.wgsl:2628-2641),
// one per tile of 64 threads; each tile's sum for all its threads.
template <class T>
__device__ __forceinline__ T tree64x4(T* s, T v) {
    const int lane = (int)(threadIdx.x & 63u), base = (int)(threadIdx.x & ~63u);
    s[threadIdx.x] = v;
    __syncthreads();
    for (int h = 32; h > 0; h >>= 1) {
        if (lane < h) s[base + lane] = s[base + lane] + s[base + lane + h];
        __syncthreads();
    }
    T r = s[base];
    __syncthreads();
    return r;
}

// sumBlocks (fluid.wgsl:2645-2661) by a 256-thread CTA, component comp of 2
// of the active blocks' partials: thread li adds the partials of blocks li,
// li + 256, ... in that order (loaded ahead in coalesced batches of 16, the
// adds kept in order), then the tree over the 256.
template <class T>
__device__ T sumBlocks256(const W& w, const T* part, int comp, T* s) {
    const uint32_t B = w.D.B;
    const uint32_t* state = w.D.blocks + B;
    const uint32_t li = threadIdx.x;
    T acc = T(0);
    for (uint32_t k0 = li; k0 < B; k0 += 256u * 16u) {
        T v[16];
        uint32_t st[16];
#pragma unroll
        for (int u = 0; u < 16; u++) {
            const uint32_t k = k0 + 256u * (uint32_t)u;
            st[u] = k < B ? __ldcg(&state[k]) : 0u;
            v[u] = k < B ? __ldcg(&part[(uint32_t)comp * B + k]) : T(0);
        }
#pragma unroll
        for (int u = 0; u < 16; u++)
            if ((st[u] & ACTIVE) != 0u) acc = acc + v[u];
    }
    s[li] = acc;
    __syncthreads();
    for (int h = 128; h > 32; h >>= 1) {
        if ((int)li < h) s[li] = s[li] + s[li + h];
        __syncthreads();
    }
    if (li < 32u) {
        T v = s[li] + s[li + 32u];
#pragma unroll
        for (int h = 16; h > 0; h >>= 1) v = v + __shfl_down_sync(0xffffffffu, v, h);
        if (li == 0u) s[0] = v;
    }
    __syncthreads();
    T r = s[0];
    __syncthreads();
    return r;
}

// Whether this CTA counted the last of `total` tiles: a threadfence
// reduction's test.  The partials of the counted tiles were written by the
// tiles' first threads (threadIdx.x % 64 == 0), each with no fence of its
// own: those threads fence here, once for all the tiles of the run, before
// the count.
__device__ bool lastOf4(uint32_t* counter, uint32_t inc, uint32_t total) {
    __shared__ int last;
    if ((threadIdx.x & 63u) == 0u) __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t old = atomicAdd(counter, inc);
        last = old + inc == total ? 1 : 0;
        if (last) {
            *counter = 0u;
            __threadfence();
        }
    }
    __syncthreads();
    return last != 0;
}

// Whether a CTA's run over a list ends its share of a world at item g (the
// run's last item, or the next item is another world's): where it counts
// the tiles it finished, one atomic per world a CTA instead of one per item.
__device__ __forceinline__ bool worldRunEnds(const Batch& Bt, uint32_t list, uint32_t g, uint32_t e, uint32_t it) {
    if (g + 1u >= e) return true;
    return ((uint64_t)Bt.item(list, g + 1u) >> Bt.lbits) != ((uint64_t)it >> Bt.lbits);
}

// At the end of a world's run: counts the CTA's pending tiles of that world;
// true in the CTA that counted the world's last tile.
__device__ __forceinline__ bool flushTiles(const Batch& Bt, uint32_t g, uint32_t e, uint32_t it, uint32_t& pend,
                                           uint32_t* counter, uint32_t total) {
    if (!worldRunEnds(Bt, L_ACT4, g, e, it)) return false;
    const uint32_t inc = pend;
    pend = 0u;
    return lastOf4(counter, inc, total);
}

__device__ __forceinline__ I2 tileCell(const W& w, uint32_t wid) {
    I2 b = w.activeBlock(wid);
    return I2{b.x * BLOCK + (int)(threadIdx.x & 7u), b.y * BLOCK + (int)((threadIdx.x >> 3) & 7u)};
}

// An item's world: its descriptor D, fast scratch F, accessors w, unit j,
// from the CTA's copy of the world (every thread of the CTA, each item in
// turn; the kernel declares `__shared__ WorldCopy wc_;`) or (FAST_ITEM_G)
// from the world table.
#define FAST_ITEM(Bt, it, D, F, w, j)            \
    const World& Wd_##it = src.get((Bt), (it), wc_); \
    const Dev& D = Wd_##it.D;                    \
    const FastW& F = Wd_##it.S;                  \
    const W w(D);                                \
    const uint32_t j = (Bt).unit(it)
#define FAST_ITEM_G(Bt, it, D, F, w, j)          \
    const World& Wd_##it = (Bt).world(it);       \
    const Dev& D = Wd_##it.D;                    \
    const FastW& F = Wd_##it.S;                  \
    const W w(D);                                \
    const uint32_t j = (Bt).unit(it)

// ================================================================ set-up

// cgStart, cgResidual, cgPrepare (fluid.wgsl:2665-2732) into the scratch,
// the cells' coefficients worked out (four tiles a 256-thread CTA, a world's
// group of four active blocks an item; the CTA that counts a world's last
// tile sums its ||b||^2), and the partial sums of the blocks not worked on
// zeroed (the invariant; a block may have dropped out in any way since: as
// the list of the retired says, or by a host's hand in the blocks' words).
template <bool ONE, bool BODIES>
__global__ void __launch_bounds__(256) k_fSetup(Batch Bt, const __grid_constant__ WorldSrc<ONE> src) {
    __shared__ WorldCopy wc_;
    if (!ONE) worldCopyInit(wc_);
    __shared__ double s64[256];
    uint32_t pend_ = 0;  // tiles finished of the current world, not yet counted
    FOR_ITEMS(Bt, L_ACT4, it) {
        FAST_ITEM(Bt, it, D, F, w, g);
        const uint32_t na = w.activeCount();
        const bool tol = D.st->tol_mode != 0u;
        const Fine& Z = F.Z;
        const uint32_t wid = g * 4u + (threadIdx.x >> 6);
        const bool valid = wid < na;
        double b2 = 0.0;
        I2 c{-1, -1};
        if (valid) c = tileCell(w, wid);
        if (valid && w.inWorld(c)) {
            const uint32_t i = w.cellIndex(c);
            const float4 gc = w.f4(2u * i), dr = w.f4(2u * i + 1u);
            const float rho = gc.z;
            Z.rho[i] = rho;
            F.X[i] = gc.x;
            F.P[i] = 0.0f;
            F.Q[i] = 0.0f;
            Z.pot[i] = make_float2(0.0f, dr.x);
            Z.rim[i] = make_float2(0.0f, dr.x);
            Z.ry[i] = dr.y;
            float bb[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            float R = 0.0f;
            uint32_t mask = 0;
            if (rho > 0.0f) {
                mask = FM_LIQUID;
                const float share = w.densityAt(c);
                float sx = 0.0f, dg = 0.0f;
                for (int d = 0; d < 4; d++) {
                    I2 n = beside(c, d);
                    if (!w.inWorld(n)) continue;
                    float4 gn = w.f4(2u * w.cellIndex(n));
                    float r = gn.z;
                    if (r < 0.0f) continue;
                    float beta = fineBeta(rho, r, share, w.densityAt(n));
                    bb[d] = beta;
                    if (r > 0.0f) mask |= 1u << d;
                    // the stencil over the warm pressure (cgResidual runs before cgPrepare)
                    sx = sx + beta * gn.x;
                    dg = dg + beta;
                }
                const float pinv = (vld(w.gwp(i, G_REGION)) == i) ? PIN : 0.0f;
                if (pinv > 0.0f) mask |= FM_PIN;
                float res = gc.y - (sx - (dg + pinv) * gc.x) / 1.0f;
                float coupled = 0.0f;
                if (BODIES) {
                    coupled = couplingAt(w, c, PUSH_X);
                    for (int d = 0; d < 4; d++)
                        if (rigidAt(w, beside(c, d)) != NONE) mask |= FM_BODY;
                }
                R = -res - coupled;
                double bd = (double)gc.y;
                b2 = bd * bd;
            }
            Z.b[i] = make_float4(bb[0], bb[1], bb[2], bb[3]);
            if (Bt.mixed) {
                // the smoother's copies of the coefficients (the mixed form)
                __half2* h = reinterpret_cast<__half2*>(F.H[0].base) + 2u * (size_t)i;
                h[0] = __floats2half2_rn(bb[0], bb[1]);
                h[1] = __floats2half2_rn(bb[2], bb[3]);
            }
            Z.mask[i] = (uint8_t)mask;
            F.R[i] = R;
        }
        if (tol) {
            double v = tree64x4(s64, b2);
            if (valid && (threadIdx.x & 63u) == 0u) {
                D.norm64[w.blockIndex(w.activeBlock(wid))] = v;
            }
            pend_ += min(4u, na - g * 4u);
            if (flushTiles(Bt, g_it, e_it, it, pend_, &D.st->fdone[0], na)) {
                double bn = sumBlocks256(w, D.norm64, 0, s64);
                if (threadIdx.x == 0) {
                    D.st->bnorm2 = bn;
                    D.st->rel = 1.0;
                }
            }
        }
    }
    const uint32_t nb = Bt.n(L_WB);
    for (uint32_t t = blockIdx.x * 256u + threadIdx.x; t < nb; t += gridDim.x * 256u) {
        const uint32_t it = Bt.item(L_WB, t);
        const World& Wd = src.getG(Bt, it);
        const uint32_t n = Bt.unit(it);
        if ((Wd.D.blocks[W(Wd.D).stateSlot(n)] & ACTIVE) == 0u) zeroPartials(Wd.D, Wd.S, n);
    }
}

// The level-0 arrays neighbours read, zeroed in the blocks not worked on
// (the invariant), for worlds whose scratch is lent by a pool for the step: a
// CTA per block of the world.
__global__ void k_fZeroIdle(Batch Bt) {
    FOR_ITEMS(Bt, L_WB, it) {
        FAST_ITEM_G(Bt, it, D, F, w, n);
        if (D.st->book != 0u || (D.blocks[w.stateSlot(n)] & ACTIVE) != 0u) continue;
        for (uint32_t t = threadIdx.x; t < 64u; t += blockDim.x) {
            const I2 bq_ = w.blockAt(n);
            I2 c{bq_.x * BLOCK + (int)(t & 7u), bq_.y * BLOCK + (int)(t >> 3)};
            if (!w.inWorld(c)) continue;
            const uint32_t i = w.cellIndex(c);
            zeroFine(F, i);
        }
    }
}

// Zeroes the level-0 arrays the neighbours read (after an upload).
__global__ void k_fZero(Dev D, FastW F) {
    const uint32_t C = D.C;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < C; i += gridDim.x * blockDim.x) {
        zeroFine(F, i);
    }
}

// ================================================================ level storage

// A coarse level's arrays as stored, the operator (density, stencil
// coefficients) in T: f32 (the plain precision) or binary16 (the mixed
// form); values are read into and worked in f32.  The potentials,
// right-hand sides and way-up potentials of a level whose operator is stored
// as T: f32 with an f32 operator; bf16 (8 bits of mantissa, f32's range, so
// no scaling as a residual shrinks) with the mixed form's binary16 operator.
// Both are stored in the level's f32 arrays (a bf16 array fills the first
// half of one).
template <class T>
struct PotOf {
    using type = float;
};
template <>
struct PotOf<__half> {
    using type = __nv_bfloat16;
};
__device__ __forceinline__ float ld(const float* p) { return *p; }
__device__ __forceinline__ float ld(const __half* p) { return __half2float(*p); }
__device__ __forceinline__ float ld(const __nv_bfloat16* p) { return __bfloat162float(*p); }
__device__ __forceinline__ void st(float* p, float v) { *p = v; }
__device__ __forceinline__ void st(__half* p, float v) { *p = __float2half_rn(v); }
__device__ __forceinline__ void st(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }

// A cell's coefficients' sum, its diagonal.  In binary16 of the rounded
// coefficients, so the rounded operator keeps its diagonal equal to the sum
// of its off-diagonals (a separately rounded diagonal could fall below it
// and make a region with no free surface indefinite).
__device__ __forceinline__ float diagOf(float4 b) { return ((b.x + b.y) + b.z) + b.w; }

// Levels 1 down as the form stores them: potentials and right-hand sides of
// PotOf<T>, densities and coefficients of T.
template <class T>
struct LRef {
    using P = typename PotOf<T>::type;
    P *px, *py, *rx, *ry;
    T *rho, *b0, *b1, *b2, *b3;
    __device__ __forceinline__ float2 pot(uint32_t k) const { return make_float2(ld(px + k), ld(py + k)); }
    __device__ __forceinline__ float2 rhs(uint32_t k) const { return make_float2(ld(rx + k), ld(ry + k)); }
    __device__ __forceinline__ float4 coef(uint32_t k) const {
        return make_float4(ld(b0 + k), ld(b1 + k), ld(b2 + k), ld(b3 + k));
    }
    __device__ __forceinline__ float dens(uint32_t k) const { return ld(rho + k); }
    __device__ __forceinline__ float pin(uint32_t) const { return 0.0f; }
    __device__ __forceinline__ void flags(uint32_t k, bool* liquid, float* pinv) const {
        *liquid = dens(k) > 0.0f;
        *pinv = 0.0f;
    }
};
template <class T>
__device__ __forceinline__ LRef<T> lref(const FastW& F, uint32_t l);
template <>
__device__ __forceinline__ LRef<float> lref<float>(const FastW& F, uint32_t l) {
    const Lvl& V = F.L[l];
    return LRef<float>{V.px, V.py, V.rx, V.ry, V.rho, V.b0, V.b1, V.b2, V.b3};
}
template <>
__device__ __forceinline__ LRef<__half> lref<__half>(const FastW& F, uint32_t l) {
    const Lvl& V = F.L[l];
    __half* b = F.H[l].base;
    const uint32_t n = F.H[l].n;
    using P = __nv_bfloat16;
    return LRef<__half>{reinterpret_cast<P*>(V.px), reinterpret_cast<P*>(V.py), reinterpret_cast<P*>(V.rx),
                        reinterpret_cast<P*>(V.ry), b, b + n, b + 2u * n, b + 3u * n, b + 4u * n};
}
// Level 0 as the form's smoother reads it: all f32, or (the mixed form) its
// coefficients from their binary16 copies (the CG's A p keeps the f32 ones).
__device__ __forceinline__ float4 fineCoef(const FastW& F, uint32_t i, float) { return F.Z.b[i]; }
__device__ __forceinline__ float4 fineCoef(const FastW& F, uint32_t i, __half) {
    const uint2 q = reinterpret_cast<const uint2*>(F.H[0].base)[i];
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&q.x));
    const float2 c = __half22float2(*reinterpret_cast<const __half2*>(&q.y));
    return make_float4(a.x, a.y, c.x, c.y);
}
template <class T>
struct LRef0 {
    const FastW& F;
    __device__ __forceinline__ float2 pot(uint32_t k) const { return F.Z.pot[k]; }
    __device__ __forceinline__ float2 rhs(uint32_t k) const { return make_float2(-F.R[k], F.Z.ry[k]); }
    __device__ __forceinline__ float4 coef(uint32_t k) const { return fineCoef(F, k, T()); }
    __device__ __forceinline__ float dens(uint32_t k) const { return F.Z.rho[k]; }
    __device__ __forceinline__ float pin(uint32_t k) const { return (F.Z.mask[k] & FM_PIN) != 0u ? PIN : 0.0f; }
    __device__ __forceinline__ void flags(uint32_t k, bool* liquid, float* pinv) const {
        const uint32_t m = F.Z.mask[k];
        *liquid = (m & FM_LIQUID) != 0u;
        *pinv = (m & FM_PIN) != 0u ? PIN : 0.0f;
    }
};
// Level l's way-up potentials (l >= 1) as a level of operator T stores them.
template <class T>
__device__ __forceinline__ typename PotOf<T>::type* upx(const FastW& F, uint32_t l) {
    return reinterpret_cast<typename PotOf<T>::type*>(F.L[l].ux);
}
template <class T>
__device__ __forceinline__ typename PotOf<T>::type* upy(const FastW& F, uint32_t l) {
    return reinterpret_cast<typename PotOf<T>::type*>(F.L[l].uy);
}

// ================================================================ relaxation

__device__ I2 tileBlockF(const W& w, uint32_t wid, int shift) {
    if (wid < w.activeCount()) return w.activeBlock(wid);
    int wide = (int)w.D.BW, high = (int)w.D.BH;
    int j = (int)wid - (int)w.D.B;
    if (shift == 0 || j < 0 || j > high + wide) return I2{-1, -1};
    return j <= high ? I2{wide, j} : I2{j - high - 1, high};
}

// mixf(a, b, 1): a 0 + b, its product exact, so one fused operation rounds
// as the two do.
__device__ __forceinline__ float mixed1(float a, float b) {
    static_assert(SMOOTH_OMEGA == 1.0f, "the smoother's relaxation factor");
    return __fmaf_rn(a, 0.0f, b);
}

// relaxTile (fluid.wgsl:2109-2182) over the scratch, from the rim snapshot.
// A warp a tile (four a CTA, each warp its own run of the list): lane l
// holds the red and the black cell of quarter l % 4 of row l / 4, so every
// lane works in every sweep and a sweep ends at a warp barrier; and it loads
// one of the 32 cells around the tile (the stencil reads no corner).  Within
// a colour the cells are independent, so each keeps the reference's
// arithmetic and order.  Bound by its instructions: 11 loads a lane and 8
// sweeps of two divisions each; the tile's potentials lie in pairs, rows 12
// pairs apart, so a half-warp's reads of a sweep touch each bank once.  With
// a float an array (38 loads a lane, the sweeps reading x and y apart) it
// took 17 us on the 1024x1024 world and 84 us on the 2048x2048 column.
// `second`: the iteration's relaxation after the V-cycle, on the other
// tiling from the first (each world's first tiling is its step's).
constexpr int RXS = RIM + 2;
template <class T>
__device__ __forceinline__ void relaxTile(const Dev& D, const FastW& F, const W& w, uint32_t na, uint32_t j, int shift,
                                          float2* sp) {
    const uint32_t lane = threadIdx.x & 31u;
    const int ly = (int)(lane >> 2), q = (int)(lane & 3u);
    // the lane's cell around the tile: the left and right columns, the rows
    // above and below, 8 lanes each
    const int side = (int)(lane >> 3), along = (int)(lane & 7u);
    const int rx_ = side == 0 ? -1 : side == 1 ? BLOCK : along, ry_ = side == 2 ? -1 : side == 3 ? BLOCK : along;
    const Fine& Z = F.Z;
    const uint32_t wid = j < na ? j : D.B + (j - na);
    const I2 b = tileBlockF(w, wid, shift);
    const int ox = b.x * BLOCK - shift, oy = b.y * BLOCK - shift;
    if (b.x < 0 || ox >= D.W || oy >= D.H) return;
    const uint32_t states = w.statesOf(I2{ox / BLOCK, oy / BLOCK}, I2{(ox + BLOCK - 1) / BLOCK, (oy + BLOCK - 1) / BLOCK});
    // the lane's two cells and its cell around the tile, all loads issued
    // together (and before the tile's state is known)
    const int p0 = (ox + oy + ly) & 1;
    int t[2];
    uint32_t idx[2], mk[2];
    float R[2], ry[2];
    float4 bb[2];
    float2 v[2];
#pragma unroll
    for (int c = 0; c < 2; c++) {
        const int lx = 2 * q + (c == 0 ? p0 : 1 - p0);
        const I2 me{ox + lx, oy + ly};
        const bool in = w.inWorld(me);
        t[c] = (ly + 1) * RXS + lx + 1;
        idx[c] = in ? w.cellIndex(me) : 0u;
        mk[c] = in ? Z.mask[idx[c]] : 0u;
        R[c] = F.R[idx[c]];
        ry[c] = Z.ry[idx[c]];
        bb[c] = fineCoef(F, idx[c], T());
        v[c] = in ? Z.rim[idx[c]] : make_float2(0.0f, 0.0f);
    }
    const I2 rc{ox + rx_, oy + ry_};
    const float2 around = w.inWorld(rc) ? Z.rim[w.cellIndex(rc)] : make_float2(0.0f, 0.0f);
    if ((states & HAS_FLUID) == 0u) return;
    float dx[2], dy[2];
    bool solving[2], visc[2];
#pragma unroll
    for (int c = 0; c < 2; c++) {
        const float dg = diagOf(bb[c]);
        dx[c] = dg + ((mk[c] & FM_PIN) != 0u ? PIN : 0.0f);
        dy[c] = fmaxf(dg, 1e-30f);
        solving[c] = (mk[c] & FM_LIQUID) != 0u && dx[c] > 0.0f;
        visc[c] = dg > 0.0f;
        sp[t[c]] = v[c];
    }
    sp[(ry_ + 1) * RXS + rx_ + 1] = around;
    __syncwarp();
    // (a loop, not 8 sweeps in a row: its instructions are fetched once)
#pragma unroll 1
    for (int pair = 0; pair < SWEEPS; pair++) {
#pragma unroll
        for (int c = 0; c < 2; c++) {
            if (solving[c]) {
                const float2* s = sp + t[c];
                const float2 l = s[-1], r = s[1], u = s[-RXS], d = s[RXS];
                const float sx = bb[c].x * l.x + bb[c].y * r.x + bb[c].z * u.x + bb[c].w * d.x;
                const float sy = bb[c].x * l.y + bb[c].y * r.y + bb[c].z * u.y + bb[c].w * d.y;
                // the right-hand side is -R
                v[c].x = mixed1(v[c].x, (sx + R[c]) / dx[c]);
                const float ny = mixed1(v[c].y, (sy - ry[c]) / dy[c]);
                if (visc[c]) v[c].y = ny;
                sp[t[c]] = v[c];
            }
            __syncwarp();
        }
    }
#pragma unroll
    for (int c = 0; c < 2; c++)
        if (solving[c]) Z.pot[idx[c]] = v[c];
}

template <bool ONE, class T>
__global__ void __launch_bounds__(128) k_fRelax(Batch Bt, const __grid_constant__ WorldSrc<ONE> src, int second) {
    __shared__ float2 tp[4][RIM * RXS];
    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t n = Bt.n(L_RELAX);
    const uint32_t warps = gridDim.x * 4u, per = (n + warps - 1u) / warps;
    const uint32_t first = (blockIdx.x * 4u + warp) * per, last = min(first + per, n);
#pragma unroll 1
    for (uint32_t g = first; g < last; g++) {
        const uint32_t it = Bt.item(L_RELAX, g);
        const World& Wd = src.getG(Bt, it);
        const Dev& D = Wd.D;
        const W w(D);
        if (D.st->cont == 0u) continue;
        const int shift = ((D.st->shift_first ^ (uint32_t)second) & 1u) ? BLOCK / 2 : 0;
        relaxTile<T>(D, Wd.S, w, w.activeCount(), Bt.unit(it), shift, tp[warp]);
    }
}

// ================================================================ the levels

// residualAt (fluid.wgsl:2306-2315) of a cell from its coefficients, its
// potentials p, its neighbours' l, r, u, d, its right-hand side and pin.  The
// division by h2, a power of two, is the multiplication by its exact
// inverse: the same real number rounded once either way, so the same bits.
__device__ __forceinline__ V2 residualOf(float4 b, float2 p, float2 l, float2 r, float2 u, float2 d, float2 rhs, float pin,
                                         float inv_h2) {
    const float sx = (((0.0f + b.x * l.x) + b.y * r.x) + b.z * u.x) + b.w * d.x;
    const float sy = (((0.0f + b.x * l.y) + b.y * r.y) + b.z * u.y) + b.w * d.y;
    const float dg = diagOf(b);
    return V2{rhs.x - (sx - (dg + pin) * p.x) * inv_h2, rhs.y - (sy - (dg + 0.0f) * p.y) * inv_h2};
}

// restrictLevel's values of level-l cell (cx, cy) from level l - 1, stored
// as VT reads it (fluid.wgsl:2342-2377): the density and, with `res`, the
// restricted residuals; all 0 in a block not worked on.  The four finer
// cells' words and the 12 potentials their stencils share are all loaded
// before any is used (coordinates clamped onto the level, as the stencil's
// neighbours are onto their cell; a cell not liquid has its residual worked
// and dropped), so their loads are in flight together; the sums then take
// the liquid cells in the reference's order.
template <class VT>
__device__ __forceinline__ void restrictedFrom(const Dev& D, const W& w, uint32_t l, const VT& U, int cx, int cy, bool res,
                                               float& rho_o, float& rx_o, float& ry_o) {
    const int span = 1 << l;
    if (span <= BLOCK) {
        I2 b{cx * span / BLOCK, cy * span / BLOCK};
        if (w.inBlocks(b) && (D.blocks[w.stateSlot(w.blockIndex(b))] & ACTIVE) == 0u) {
            rho_o = 0.0f;
            rx_o = 0.0f;
            ry_o = 0.0f;
            return;
        }
    }
    const int uw = (int)D.level_w[l - 1], uh = (int)D.level_h[l - 1];
    const int x0 = 2 * cx, y0 = 2 * cy;
    const bool in_x = x0 + 1 < uw, in_y = y0 + 1 < uh;  // rhoAt outside the level: -1
    const uint32_t xs[4] = {(uint32_t)max(x0 - 1, 0), (uint32_t)x0, (uint32_t)min(x0 + 1, uw - 1), (uint32_t)min(x0 + 2, uw - 1)};
    const uint32_t ys[4] = {(uint32_t)max(y0 - 1, 0) * (uint32_t)uw, (uint32_t)y0 * (uint32_t)uw,
                            (uint32_t)min(y0 + 1, uh - 1) * (uint32_t)uw, (uint32_t)min(y0 + 2, uh - 1) * (uint32_t)uw};
    float rq[4];
    V2 eq[4];
#pragma unroll
    for (int q = 0; q < 4; q++) rq[q] = U.dens(ys[1 + (q >> 1)] + xs[1 + (q & 1)]);
    if (res) {
        const float inv_h2 = 1.0f / (float)(1u << (2u * (l - 1u)));
        float2 p[4][4];  // [row][column], corners not read
        float4 bq[4];
        float2 hq[4];
        float pq[4];
#pragma unroll
        for (int y = 0; y < 4; y++)
#pragma unroll
            for (int x = 0; x < 4; x++)
                if ((x == 1 || x == 2) || (y == 1 || y == 2)) p[y][x] = U.pot(ys[y] + xs[x]);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const uint32_t k = ys[1 + (q >> 1)] + xs[1 + (q & 1)];
            bq[q] = U.coef(k);
            hq[q] = U.rhs(k);
            pq[q] = U.pin(k);
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int x = 1 + (q & 1), y = 1 + (q >> 1);
            eq[q] = residualOf(bq[q], p[y][x], p[y][x - 1], p[y][x + 1], p[y - 1][x], p[y + 1][x], hq[q], pq[q], inv_h2);
        }
    }
    float fluid = 0.0f, sum = 0.0f, rx = 0.0f, ry = 0.0f;
    bool air = false;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        if ((!in_x && (q & 1)) || (!in_y && (q >> 1))) continue;
        const float rho = rq[q];
        if (rho == 0.0f) air = true;
        else if (rho > 0.0f) {
            fluid = fluid + 1.0f;
            sum = sum + rho;
            if (res) {
                rx = rx + eq[q].x;
                ry = ry + eq[q].y;
            }
        }
    }
    const float rho = air ? 0.0f : (fluid > 0.0f ? sum / fluid : -1.0f);
    rho_o = rho;
    rx_o = rho > 0.0f ? rx * 0.25f : 0.0f;
    ry_o = rho > 0.0f ? ry * 0.25f : 0.0f;
}

// The restricted residuals alone of a liquid level-l cell (its density, like
// every level's densities and coefficients, is the step's first
// iteration's): its finer cells are liquid or obstacles.
template <class VT>
__device__ __forceinline__ V2 residualsFrom(const Dev& D, uint32_t l, const VT& U, int cx, int cy) {
    const int uw = (int)D.level_w[l - 1], uh = (int)D.level_h[l - 1];
    const int x0 = 2 * cx, y0 = 2 * cy;
    const bool in_x = x0 + 1 < uw, in_y = y0 + 1 < uh;
    const uint32_t xs[4] = {(uint32_t)max(x0 - 1, 0), (uint32_t)x0, (uint32_t)min(x0 + 1, uw - 1), (uint32_t)min(x0 + 2, uw - 1)};
    const uint32_t ys[4] = {(uint32_t)max(y0 - 1, 0) * (uint32_t)uw, (uint32_t)y0 * (uint32_t)uw,
                            (uint32_t)min(y0 + 1, uh - 1) * (uint32_t)uw, (uint32_t)min(y0 + 2, uh - 1) * (uint32_t)uw};
    const float inv_h2 = 1.0f / (float)(1u << (2u * (l - 1u)));
    float2 p[4][4];  // [row][column], corners not read
    float4 bq[4];
    float2 hq[4];
    float pq[4];
    bool liquid[4];
#pragma unroll
    for (int y = 0; y < 4; y++)
#pragma unroll
        for (int x = 0; x < 4; x++)
            if ((x == 1 || x == 2) || (y == 1 || y == 2)) p[y][x] = U.pot(ys[y] + xs[x]);
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const uint32_t k = ys[1 + (q >> 1)] + xs[1 + (q & 1)];
        bq[q] = U.coef(k);
        hq[q] = U.rhs(k);
        U.flags(k, &liquid[q], &pq[q]);
    }
    float rx = 0.0f, ry = 0.0f;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        if ((!in_x && (q & 1)) || (!in_y && (q >> 1)) || !liquid[q]) continue;
        const int x = 1 + (q & 1), y = 1 + (q >> 1);
        const V2 e = residualOf(bq[q], p[y][x], p[y][x - 1], p[y][x + 1], p[y - 1][x], p[y + 1][x], hq[q], pq[q], inv_h2);
        rx = rx + e.x;
        ry = ry + e.y;
    }
    return V2{rx * 0.25f, ry * 0.25f};
}
template <class T, bool FINE>
__device__ __forceinline__ V2 residualsAt(const Dev& D, const FastW& F, uint32_t l, int cx, int cy) {
    if (FINE) return residualsFrom(D, l, LRef0<T>{F}, cx, cy);
    return residualsFrom(D, l, lref<T>(F, l - 1u), cx, cy);
}

// restrictedFrom for level l of a form whose levels store operator T: from
// level 0 as its smoother reads it (FINE: l is 1), or from level l - 1.
template <class T, bool FINE>
__device__ __forceinline__ void restrictedAt(const Dev& D, const FastW& F, const W& w, uint32_t l, int cx, int cy,
                                             bool res, float& rho_o, float& rx_o, float& ry_o) {
    if (FINE) restrictedFrom(D, w, l, LRef0<T>{F}, cx, cy, res, rho_o, rx_o, ry_o);
    else restrictedFrom(D, w, l, lref<T>(F, l - 1u), cx, cy, res, rho_o, rx_o, ry_o);
}

// One coarse cell of restrictLevel, level l from l - 1 (FINE: level 1 from
// level 0) with the levels stored as T: the cell's values, its potentials
// zeroed.
template <class T, bool FINE, bool EAGER>
__device__ void restrictCell(const Dev& D, const FastW& F, const W& w, uint32_t l, uint32_t j, bool first) {
    const int lw = (int)D.level_w[l];
    const LRef<T> V = lref<T>(F, l);
    if (!first) {
        // only a liquid cell's right-hand sides have changed
        const float rho = V.dens(j);
        if (!EAGER && !(rho > 0.0f)) return;
        const V2 r = residualsAt<T, FINE>(D, F, l, (int)(j % (uint32_t)lw), (int)(j / (uint32_t)lw));
        if (EAGER && !(rho > 0.0f)) return;
        st(V.rx + j, r.x);
        st(V.ry + j, r.y);
        return;
    }
    float rho, rx, ry;
    restrictedAt<T, FINE>(D, F, w, l, (int)(j % (uint32_t)lw), (int)(j / (uint32_t)lw), true, rho, rx, ry);
    st(V.px + j, 0.0f);
    st(V.py + j, 0.0f);
    st(V.rx + j, rx);
    st(V.ry + j, ry);
    st(V.rho + j, rho);
}

// prolonged (fluid.wgsl:2478-2497) from level l + 1's arrays.  The four
// coarse cells' words are loaded before any is used (a cell past the
// level's edge reads a clamped one and is left out), then weighed in the
// reference's order.
template <class T, class P>
__device__ __forceinline__ V2 prolongedFrom(const T* rho, const P* px, const P* py, int lw, int lh, int cx, int cy) {
    const int kx = cx / 2, ky = cy / 2;
    const int sx = (cx & 1) == 1 ? 1 : -1, sy = (cy & 1) == 1 ? 1 : -1;
    const int ox[4] = {0, sx, 0, sx}, oy[4] = {0, 0, sy, sy};
    const float wt[4] = {9.0f, 3.0f, 3.0f, 1.0f};
    float rq[4], xq[4], yq[4];
    bool inq[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int ax_ = kx + ox[q], ay_ = ky + oy[q];
        inq[q] = !(ax_ < 0 || ay_ < 0 || ax_ >= lw || ay_ >= lh);
        const uint32_t k = inq[q] ? (uint32_t)ay_ * (uint32_t)lw + (uint32_t)ax_ : 0u;
        rq[q] = ld(rho + k);
        xq[q] = ld(px + k);
        yq[q] = ld(py + k);
    }
    float ax = 0.0f, ay = 0.0f, weight = 0.0f;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        if (!inq[q]) continue;
        const float r = rq[q];
        if (r < 0.0f) continue;
        weight = weight + wt[q];
        if (r > 0.0f) {
            ax = ax + wt[q] * xq[q];
            ay = ay + wt[q] * yq[q];
        }
    }
    const float ww = fmaxf(weight, 1e-6f);
    return V2{ax / ww, ay / ww};
}

// ---------------------------------------------------------------- level tiles
//
// The levels above the coarse kernel's, a 16x16 tile of level l a 256-thread
// CTA, each pass of one level in one kernel: on the way down the tile's
// restriction and both colours of smoothing, on the way up its
// prolongation and both colours.  A tile works a ring of 2 cells around
// itself again (its neighbours' work, the same arithmetic on the same
// inputs, so the same bits): the red sweep on the ring of 1 reads the ring
// of 2, the black sweep on the tile reads the ring of 1.  Shared-memory
// arrays are 20 x 20, tile cell (0, 0) at (2, 2).

constexpr int LT = 16, LR = LT + 4, LRR = LR * LR;

__device__ __forceinline__ int lsi(int ix, int iy) { return (iy + 2) * LR + (ix + 2); }

// The shared index of neighbour d of tile cell (ix, iy) at level cell
// (cx, cy): clamped onto the cell past the level's edge, as nbr.
__device__ __forceinline__ int lsn(int ix, int iy, int cx, int cy, int lw, int lh, int d) {
    if (!nbrIn(cx, cy, lw, lh, d)) return lsi(ix, iy);
    switch (d) {
    case 0: return lsi(ix - 1, iy);
    case 1: return lsi(ix + 1, iy);
    case 2: return lsi(ix, iy - 1);
    default: return lsi(ix, iy + 1);
    }
}

// A value as a level of T stores it and reads it back.
__device__ __forceinline__ float asStored(float v, float) { return v; }
__device__ __forceinline__ float asStored(float v, __half) { return __half2float(__float2half_rn(v)); }

struct LevelTile {
    float rho[LRR], px[LRR], py[LRR], rx[LRR], ry[LRR], b[4][LRR], dg[LRR];
};

// One colour's sweep of smoothAt (fluid.wgsl:2318-2334) over tile cell
// (ix, iy) held in the tile's arrays.
__device__ __forceinline__ void tileSweepCell(LevelTile& t, int ix, int iy, int cx, int cy, int lw, int lh, float h2) {
    const int i = lsi(ix, iy);
    if (t.rho[i] <= 0.0f) return;
    const float dg = t.dg[i];
    if (dg <= 0.0f) return;
    float sx = 0.0f, sy = 0.0f;
#pragma unroll
    for (int d = 0; d < 4; d++) {
        const int n = lsn(ix, iy, cx, cy, lw, lh, d);
        sx = sx + t.b[d][i] * t.px[n];
        sy = sy + t.b[d][i] * t.py[n];
    }
    t.px[i] = mixf(t.px[i], (sx - h2 * t.rx[i]) / dg, SMOOTH_OMEGA);
    t.py[i] = mixf(t.py[i], (sy - h2 * t.ry[i]) / dg, SMOOTH_OMEGA);
}

// The NT threads that work a tile: a CTA, or a part of one under named
// barrier `bar` (0: the CTA's own).
template <int NT>
struct Team {
    int tid, bar;
    __device__ __forceinline__ void sync() const {
        if (bar == 0) __syncthreads();
        else asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(NT) : "memory");
    }
};

// The red sweep over the tile's ring of 1, the black over the tile itself.
template <int NT>
__device__ __forceinline__ void tileSmooth(LevelTile& t, const Team<NT>& tm, int x0, int y0, int lw, int lh, float h2) {
#pragma unroll 1
    for (int k = tm.tid; k < (LT + 2) * (LT + 2); k += NT) {
        const int ix = k % (LT + 2) - 1, iy = k / (LT + 2) - 1, cx = x0 + ix, cy = y0 + iy;
        if (cx < 0 || cy < 0 || cx >= lw || cy >= lh || ((cx + cy) & 1) != 0) continue;
        tileSweepCell(t, ix, iy, cx, cy, lw, lh, h2);
    }
    tm.sync();
    if (tm.tid >= LT * LT) return;  // a wide team's threads past the tile's cells
    const int ix = tm.tid % LT, iy = tm.tid / LT, cx = x0 + ix, cy = y0 + iy;
    if (cx < lw && cy < lh && ((cx + cy) & 1) == 1) tileSweepCell(t, ix, iy, cx, cy, lw, lh, h2);
}

// Down, level l: restrictLevel, then smoothRed and smoothBlack when the
// world smooths level l (l < its coarse kernel's first level; else the
// restriction alone).  The densities and the coefficients of a level are the
// same in every iteration of a step: the first works the densities out on
// the ring of 2 and from them the coefficients of each liquid cell of the
// ring of 1, and the tile's own cells store both and whether the tile holds
// any liquid; the later ones read them back, work the residuals of liquid
// cells alone, and leave a tile without liquid as it is.  (With all of it
// worked again every time, for every tile, the down launches took 37 us of
// an iteration at 1024x1024 and 72 us on a 48-world batch.)
//
// A level of few tiles is bound by the chain of its loads, not by what it
// loads: its launches (k_fDown with 512 threads) work it all AGAIN every
// time, a round of loads (the 256x256 dam 788 us a step; reading back, first
// the tile's flag, then the density, then the rest, 809), and the one-launch
// solves of small worlds read back EAGER, loading every word a cell may need
// before the flag or the density says whether it does (a 256x256 tank with
// bodies 1371 -> 1295; on the 1024x1024 disks, where the skipped tiles and
// cells count, 4688 -> 5028, so the grid without bodies does not).
template <class T, int NT, bool FINE, bool AGAIN, bool EAGER>
__device__ __forceinline__ void downTile(const Dev& D, const FastW& F, const W& w, uint32_t l, uint32_t tile, bool first,
                                         LevelTile& t, const Team<NT>& tm) {
    const int lw = (int)D.level_w[l], lh = (int)D.level_h[l], tw = (lw + LT - 1) / LT;
    const int x0 = (int)(tile % (uint32_t)tw) * LT, y0 = (int)(tile / (uint32_t)tw) * LT;
    uint8_t* live = F.L[l].live + tile;
    if (!AGAIN && !EAGER && !first && l < F.lc && *live == 0) return;
    if (l >= F.lc) {
        const int cx = x0 + tm.tid % LT, cy = y0 + tm.tid / LT;
        if (tm.tid < LT * LT && cx < lw && cy < lh)
            restrictCell<T, FINE, EAGER>(D, F, w, l, (uint32_t)(cy * lw + cx), AGAIN || first);
        return;
    }
    const LRef<T> V = lref<T>(F, l);
    if (AGAIN || first) {
        if (first && tm.tid == 0) *live = 0;
#pragma unroll 1
        for (int k = tm.tid; k < LRR; k += NT) {
            const int ix = k % LR - 2, iy = k / LR - 2, cx = x0 + ix, cy = y0 + iy;
            float rho = -1.0f, rx = 0.0f, ry = 0.0f;
            if (cx >= 0 && cy >= 0 && cx < lw && cy < lh) {
                const bool res = ix >= -1 && iy >= -1 && ix <= LT && iy <= LT;
                restrictedAt<T, FINE>(D, F, w, l, cx, cy, res, rho, rx, ry);
            }
            t.rho[k] = asStored(rho, T());
            t.rx[k] = rx;
            t.ry[k] = ry;
            t.px[k] = 0.0f;
            t.py[k] = 0.0f;
        }
        tm.sync();
#pragma unroll 1
        for (int k = tm.tid; k < (LT + 2) * (LT + 2); k += NT) {
            const int ix = k % (LT + 2) - 1, iy = k / (LT + 2) - 1, cx = x0 + ix, cy = y0 + iy;
            if (cx < 0 || cy < 0 || cx >= lw || cy >= lh) continue;
            const int i = lsi(ix, iy);
            const float rho = t.rho[i];
            if (rho <= 0.0f) continue;
            float b[4];
#pragma unroll
            for (int d = 0; d < 4; d++) {
                b[d] = 0.0f;
                if (!nbrIn(cx, cy, lw, lh, d)) continue;
                const float r = t.rho[lsn(ix, iy, cx, cy, lw, lh, d)];
                if (r < 0.0f) continue;
                b[d] = faceBeta(rho, r);
            }
            const bool own = ix >= 0 && iy >= 0 && ix < LT && iy < LT;
            if (first && own) {
                const uint32_t j = (uint32_t)(cy * lw + cx);
                st(V.b0 + j, b[0]); st(V.b1 + j, b[1]); st(V.b2 + j, b[2]); st(V.b3 + j, b[3]);
            }
#pragma unroll
            for (int d = 0; d < 4; d++) t.b[d][i] = asStored(b[d], T());
            t.dg[i] = ((t.b[0][i] + t.b[1][i]) + t.b[2][i]) + t.b[3][i];
        }
        tm.sync();
        // (written after the barrier above, which follows the clearing)
        if (first && tm.tid < LT * LT && t.rho[lsi(tm.tid % LT, tm.tid / LT)] > 0.0f) *live = 1;
    } else {
#pragma unroll 1
        for (int k = tm.tid; k < LRR; k += NT) {
            const int ix = k % LR - 2, iy = k / LR - 2, cx = x0 + ix, cy = y0 + iy;
            float rho = -1.0f;
            if (cx >= 0 && cy >= 0 && cx < lw && cy < lh) {
                const uint32_t j = (uint32_t)(cy * lw + cx);
                rho = V.dens(j);
                if ((EAGER || rho > 0.0f) && ix >= -1 && iy >= -1 && ix <= LT && iy <= LT) {
                    const float4 b = V.coef(j);
                    const V2 r = residualsAt<T, FINE>(D, F, l, cx, cy);
                    if (!EAGER || rho > 0.0f) {
                        t.rx[k] = r.x;
                        t.ry[k] = r.y;
                        t.b[0][k] = b.x;
                        t.b[1][k] = b.y;
                        t.b[2][k] = b.z;
                        t.b[3][k] = b.w;
                        t.dg[k] = diagOf(b);
                    }
                }
            }
            t.rho[k] = rho;
            t.px[k] = 0.0f;
            t.py[k] = 0.0f;
        }
        tm.sync();
    }
    tileSmooth(t, tm, x0, y0, lw, lh, (float)(1u << (2u * l)));
    if (tm.tid < LT * LT) {
        const int ix = tm.tid % LT, iy = tm.tid / LT, cx = x0 + ix, cy = y0 + iy;
        if (cx < lw && cy < lh) {
            const uint32_t j = (uint32_t)(cy * lw + cx);
            const int i = lsi(ix, iy);
            if (AGAIN || first || t.rho[i] > 0.0f) {
                st(V.px + j, t.px[i]);
                st(V.py + j, t.py[i]);
                st(V.rx + j, t.rx[i]);
                st(V.ry + j, t.ry[i]);
            }
            if (first) st(V.rho + j, t.rho[i]);
        }
    }
    tm.sync();  // the tile's arrays are free for the next tile
}

template <bool ONE, class T, int NT, bool FINE>
__global__ void __launch_bounds__(NT, NT == 256 ? 4 : 2) k_fDown(Batch Bt, const __grid_constant__ WorldSrc<ONE> src, uint32_t l) {
    __shared__ WorldCopy wc_;
    if (!ONE) worldCopyInit(wc_);
    __shared__ LevelTile t;
    const Team<NT> tm{(int)threadIdx.x, 0};
    FOR_ITEMS(Bt, L_RES + l - 1u, it) {
        FAST_ITEM(Bt, it, D, F, w, tile);
        if (D.st->cont == 0u) continue;
        downTile<T, NT, FINE, NT == 512, false>(D, F, w, l, tile, D.st->cycle == 0u, t, tm);
    }
}

// Up, level l (< the coarse kernel's first): prolong from level l + 1
// (fluid.wgsl:2459-2497), then smoothRed and smoothBlack with the stored
// coefficients.  The way down's potentials are read from px, py (the ring
// too) and the results go to ux, uy, so no CTA reads a cell that another
// writes in the same launch; level l + 1's results are its ux, uy.
template <class T, int NT, bool EAGER>
__device__ __forceinline__ void upTile(const Dev& D, const FastW& F, uint32_t l, uint32_t tile, LevelTile& t,
                                       const Team<NT>& tm) {
    if (!EAGER && F.L[l].live[tile] == 0) return;  // no liquid: nothing to move
    const int lw = (int)D.level_w[l], lh = (int)D.level_h[l], tw = (lw + LT - 1) / LT;
    const int x0 = (int)(tile % (uint32_t)tw) * LT, y0 = (int)(tile / (uint32_t)tw) * LT;
    const LRef<T> V = lref<T>(F, l);
    const T* urho = lref<T>(F, l + 1u).rho;
    const auto* lux = upx<T>(F, l + 1u);
    const auto* luy = upy<T>(F, l + 1u);
    const int uw = (int)D.level_w[l + 1], uh = (int)D.level_h[l + 1];
#pragma unroll 1
    for (int k = tm.tid; k < LRR; k += NT) {
        const int ix = k % LR - 2, iy = k / LR - 2, cx = x0 + ix, cy = y0 + iy;
        float rho = -1.0f, px = 0.0f, py = 0.0f;
        if (cx >= 0 && cy >= 0 && cx < lw && cy < lh) {
            // every word the cell may need loaded before any is used (a
            // cell not liquid drops them)
            const uint32_t j = (uint32_t)(cy * lw + cx);
            const bool ring1 = ix >= -1 && iy >= -1 && ix <= LT && iy <= LT;
            rho = ld(V.rho + j);
            px = ld(V.px + j);
            py = ld(V.py + j);
            const V2 e = prolongedFrom(urho, lux, luy, uw, uh, cx, cy);
            float rx = 0.0f, ry = 0.0f, b0 = 0.0f, b1 = 0.0f, b2 = 0.0f, b3 = 0.0f;
            if (ring1) {
                rx = ld(V.rx + j);
                ry = ld(V.ry + j);
                b0 = ld(V.b0 + j);
                b1 = ld(V.b1 + j);
                b2 = ld(V.b2 + j);
                b3 = ld(V.b3 + j);
            }
            if (rho > 0.0f) {
                px = px + e.x;
                py = py + e.y;
                if (ring1) {
                    t.rx[k] = rx;
                    t.ry[k] = ry;
                    t.b[0][k] = b0;
                    t.b[1][k] = b1;
                    t.b[2][k] = b2;
                    t.b[3][k] = b3;
                    t.dg[k] = ((b0 + b1) + b2) + b3;
                }
            }
        }
        t.rho[k] = rho;
        t.px[k] = px;
        t.py[k] = py;
    }
    tm.sync();
    tileSmooth(t, tm, x0, y0, lw, lh, (float)(1u << (2u * l)));
    if (tm.tid < LT * LT) {
        const int ix = tm.tid % LT, iy = tm.tid / LT, cx = x0 + ix, cy = y0 + iy;
        const int i = lsi(ix, iy);
        if (cx < lw && cy < lh && t.rho[i] > 0.0f) {
            const uint32_t j = (uint32_t)(cy * lw + cx);
            st(upx<T>(F, l) + j, t.px[i]);
            st(upy<T>(F, l) + j, t.py[i]);
        }
    }
    tm.sync();
}

template <bool ONE, class T, int NT = 256>
__global__ void __launch_bounds__(NT, NT == 256 ? 4 : 2) k_fUp(Batch Bt, const __grid_constant__ WorldSrc<ONE> src, uint32_t l) {
    __shared__ WorldCopy wc_;
    if (!ONE) worldCopyInit(wc_);
    __shared__ LevelTile t;
    const Team<NT> tm{(int)threadIdx.x, 0};
    FOR_ITEMS(Bt, L_SM + l - 1u, it) {
        FAST_ITEM(Bt, it, D, F, w, tile);
        (void)w;
        if (D.st->cont == 0u) continue;
        upTile<T, NT, NT == 512>(D, F, l, tile, t, tm);
    }
}

// Named barrier `id` over `count` threads (a multiple of 32).
__device__ __forceinline__ void barSub(int id, int count) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}

// Level l (lc <= l <= levels) of the one-CTA kernel's shared memory: nine
// arrays of the level's cells from sm + off[l]: the potentials, the
// right-hand sides, the densities and the four face coefficients.
constexpr uint32_t SLV_ARRAYS = 9;
struct SLv {
    float *px, *py, *rx, *ry, *rho, *b0, *b1, *b2, *b3;
    int w, h;
    uint32_t mw;  // ceil(2^32 / w) (0 for w = 1): j / w = umulhi(j, mw) for the level's indices
};
__device__ __forceinline__ SLv slv(float* sm, const uint32_t* off, const Dev& D, uint32_t l) {
    const int n = (int)(D.level_w[l] * D.level_h[l]);
    float* p = sm + off[l];
    const uint32_t w = D.level_w[l];
    return SLv{p,         p + n,     p + 2 * n, p + 3 * n, p + 4 * n, p + 5 * n,
               p + 6 * n, p + 7 * n, p + 8 * n, (int)w, (int)D.level_h[l], w == 1u ? 0u : 0xffffffffu / w + 1u};
}
// The row of index j < 2 n of level V: j / w by a multiply-high with
// ceil(2^32 / w), exact while j w < 2^32 (the coarse kernel's levels hold at
// most 4096 cells), in place of an integer division's instruction sequence.
__device__ __forceinline__ int slvRow(const SLv& V, int j) {
    return V.w == 1 ? j : (int)__umulhi((uint32_t)j, V.mw);
}

// The face coefficients of level V's cells (smoothAt's stencil,
// fluid.wgsl:2318-2334): faceBeta to each neighbour inside the level whose
// density is not negative, else 0; all 0 for a cell that is not liquid.
__device__ void slv_coefficients(const SLv& V, int tid, int nt) {
    const int n = V.w * V.h;
#pragma unroll 1
    for (int j = tid; j < n; j += nt) {
        const int cy = slvRow(V, j), cx = j - cy * V.w;
        const float rho = V.rho[j];
        float b[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (rho > 0.0f) {
#pragma unroll
            for (int d = 0; d < 4; d++) {
                if (!nbrIn(cx, cy, V.w, V.h, d)) continue;
                const float r = V.rho[nbr((uint32_t)j, cx, cy, V.w, V.h, d)];
                if (r >= 0.0f) b[d] = faceBeta(rho, r);
            }
        }
        V.b0[j] = b[0];
        V.b1[j] = b[1];
        V.b2[j] = b[2];
        V.b3[j] = b[3];
    }
}

// The stencil's sums at liquid cell j from the stored coefficients: the
// sums of the neighbours taken in order, each beta times the neighbour's
// potential, and the betas' sum.  A neighbour the stencil skips has beta 0
// and its index clamped onto j, so adding its term changes no bit.
__device__ __forceinline__ void slv_stencil(const SLv& V, int j, int cx, int cy, float* sx, float* sy, float* dg) {
    const float b0 = V.b0[j], b1 = V.b1[j], b2 = V.b2[j], b3 = V.b3[j];
    const uint32_t n0 = nbr((uint32_t)j, cx, cy, V.w, V.h, 0), n1 = nbr((uint32_t)j, cx, cy, V.w, V.h, 1);
    const uint32_t n2 = nbr((uint32_t)j, cx, cy, V.w, V.h, 2), n3 = nbr((uint32_t)j, cx, cy, V.w, V.h, 3);
    *sx = (((0.0f + b0 * V.px[n0]) + b1 * V.px[n1]) + b2 * V.px[n2]) + b3 * V.px[n3];
    *sy = (((0.0f + b0 * V.py[n0]) + b1 * V.py[n1]) + b2 * V.py[n2]) + b3 * V.py[n3];
    *dg = (((0.0f + b0) + b1) + b2) + b3;
}

// One sweep of one colour over level V (smoothRed/Black, fluid.wgsl:2318-
// 2334, or the solve's SOR sweeps with omega): a thread per cell of that
// colour.  Of the cells 2k and 2k + 1 exactly one has each colour (in a row,
// or across a row's end when the width is odd), so pair k gives the cell.
__device__ void slv_sweep(const SLv& V, uint32_t l, int color, float omega, int tid, int nt) {
    const int n = V.w * V.h, pairs = (n + 1) / 2;
    const float h2 = (float)(1u << (2u * l));
#pragma unroll 1
    for (int k = tid; k < pairs; k += nt) {
        int j = 2 * k, cy = slvRow(V, j), cx = j - cy * V.w;
        if (((cx + cy) & 1) != color) {
            j++;
            if (++cx == V.w) {
                cx = 0;
                cy++;
            }
        }
        if (j >= n) continue;
        if (V.rho[j] <= 0.0f) continue;
        float sx, sy, dg;
        slv_stencil(V, j, cx, cy, &sx, &sy, &dg);
        if (dg <= 0.0f) continue;
        V.px[j] = mixf(V.px[j], (sx - h2 * V.rx[j]) / dg, omega);
        V.py[j] = mixf(V.py[j], (sy - h2 * V.ry[j]) / dg, omega);
    }
}

__device__ void slv_smooth(const SLv& V, uint32_t l, int tid, int nt) {
#pragma unroll 1
    for (int color = 0; color < 2; color++) {
        slv_sweep(V, l, color, SMOOTH_OMEGA, tid, nt);
        __syncthreads();
    }
}

// A coarsest-level cell of the solve, held in registers: its index, its
// four neighbours (clamped, nbr), their coefficients, the diagonal's FP64
// reciprocal (quotBy: the 80 sweeps' divisions by it), h^2 times its
// right-hand sides, and whether it is updated (a liquid cell with a
// positive diagonal, j < n).
struct SolveCell {
    uint32_t j, nb[4];
    float b[4], dg, hx, hy;
    double rd;
    int color;
    bool mine;
};
__device__ __forceinline__ SolveCell solveCell(const SLv& V, int j, int n, float h2) {
    SolveCell c;
    const int cy = slvRow(V, j), cx = j - cy * V.w;
    c.j = (uint32_t)j;
    c.color = (cx + cy) & 1;
    float r0 = -1.0f;
    c.dg = 0.0f;
    c.hx = 0.0f;
    c.hy = 0.0f;
#pragma unroll
    for (int d = 0; d < 4; d++) {
        c.b[d] = 0.0f;
        c.nb[d] = 0u;
    }
    if (j < n) {
        r0 = V.rho[j];
        c.hx = h2 * V.rx[j];
        c.hy = h2 * V.ry[j];
        c.b[0] = V.b0[j]; c.b[1] = V.b1[j]; c.b[2] = V.b2[j]; c.b[3] = V.b3[j];
#pragma unroll
        for (int d = 0; d < 4; d++) c.nb[d] = nbr((uint32_t)j, cx, cy, V.w, V.h, d);
        c.dg = (((0.0f + c.b[0]) + c.b[1]) + c.b[2]) + c.b[3];
    }
    c.mine = j < n && r0 > 0.0f && c.dg > 0.0f;
    c.rd = recipOf(c.dg);
    return c;
}
// One SOR update (omega 1.8) of a solve cell's potential v in P, h^2 times
// its right-hand side h, from its neighbours' potentials.
__device__ __forceinline__ void solveUpdate(float* P, const SolveCell& c, float h, float& v) {
    if (!c.mine) return;
    const float s = c.b[0] * P[c.nb[0]] + c.b[1] * P[c.nb[1]] + c.b[2] * P[c.nb[2]] + c.b[3] * P[c.nb[3]];
    v = mixf(v, quotBy(s - h, c.rd), OMEGA);
    P[c.j] = v;
}

// The levels from lc (in sm from offsets off[]: just loaded, or restricted
// already) down to the coarsest and back up to lc: each level's
// coefficients worked out once its densities are in place, smoothRed/Black,
// restrictLevel, solve (40 SOR sweep pairs, omega 1.8), prolong
// (fluid.wgsl:2318-2470); the result in level lc's px, py.  Every thread of
// the CTA takes part.
__device__ void coarseCore(const Dev& D, const W& w, uint32_t lc, float* sm, const uint32_t* off) {
    const uint32_t L = D.levels;
    const int tid = (int)threadIdx.x, nt = (int)blockDim.x;
#pragma unroll 1
    for (uint32_t l = lc; l <= L; l++) {
        const SLv V = slv(sm, off, D, l);
        const int n = V.w * V.h;
        if (l > lc) {
            const SLv U = slv(sm, off, D, l - 1u);
            const int span = 1 << l;
            // 1 / h^2 of level l - 1: a power of two, so the product is the
            // quotient's bits
            const float inv_h2u = 1.0f / (float)(1u << (2u * (l - 1u)));
#pragma unroll 1
            for (int j = tid; j < n; j += nt) {
                const int cy = slvRow(V, j), cx = j - cy * V.w;
                if (span <= BLOCK) {
                    I2 b{cx * span / BLOCK, cy * span / BLOCK};
                    if (w.inBlocks(b) && (D.blocks[w.stateSlot(w.blockIndex(b))] & ACTIVE) == 0u) {
                        V.px[j] = 0.0f; V.py[j] = 0.0f; V.rx[j] = 0.0f; V.ry[j] = 0.0f; V.rho[j] = 0.0f;
                        continue;
                    }
                }
                float fluid = 0.0f, sum = 0.0f, rx = 0.0f, ry = 0.0f;
                bool air = false;
                for (int q = 0; q < 4; q++) {
                    int kx = 2 * cx + (q & 1), ky = 2 * cy + (q >> 1);
                    if (kx >= U.w || ky >= U.h) continue;
                    int k = ky * U.w + kx;
                    float rho = U.rho[k];
                    if (rho == 0.0f) air = true;
                    else if (rho > 0.0f) {
                        float sx, sy, dg;
                        slv_stencil(U, k, kx, ky, &sx, &sy, &dg);
                        fluid = fluid + 1.0f;
                        sum = sum + rho;
                        rx = rx + (U.rx[k] - (sx - (dg + 0.0f) * U.px[k]) * inv_h2u);
                        ry = ry + (U.ry[k] - (sy - (dg + 0.0f) * U.py[k]) * inv_h2u);
                    }
                }
                const float rho = air ? 0.0f : (fluid > 0.0f ? sum / fluid : -1.0f);
                V.px[j] = 0.0f;
                V.py[j] = 0.0f;
                V.rx[j] = rho > 0.0f ? rx * 0.25f : 0.0f;
                V.ry[j] = rho > 0.0f ? ry * 0.25f : 0.0f;
                V.rho[j] = rho;
            }
            __syncthreads();
        }
        slv_coefficients(V, tid, nt);
        __syncthreads();
        if (l < L) slv_smooth(V, l, tid, nt);
    }
    // solve: the coarsest level (at most 512 cells).  The pressure and the
    // drift are two solves over the same coefficients: each has its own
    // warps, under its own named barrier.  Thread k of a solve's holds cells
    // 2k and 2k + 1, one of each colour (in a row, or across a row's end when
    // the width is odd), their coefficients and potentials in registers
    // across the sweeps, so every thread updates a cell each sweep.  Bound by
    // the chain of a sweep (neighbours, sum, quotient, store, barrier) 80
    // times: 9.9 us on 16x16 cells, 12.6 with both solves in a thread; the
    // quotient in f32 with two corrections is no shorter (10.6), and a warp a
    // solve with no barrier but its own spills (77).
    {
        const SLv V = slv(sm, off, D, L);
        const int n = min(V.w * V.h, (int)WIG_MG_COARSEST);
        const float h2 = (float)(1u << (2u * L));
        const int pairs = (n + 1) / 2, npair = (pairs + 31) & ~31;
        static_assert(2 * ((WIG_MG_COARSEST / 2 + 31) & ~31) <= 1024, "the two solves' threads fit the CTA");
        const int which = tid / npair, k = tid - which * npair;
        if (which < 2) {
            SolveCell c0 = solveCell(V, 2 * k, n, h2), c1 = solveCell(V, 2 * k + 1, n, h2);
            // c0 the colour-0 cell, c1 the colour-1 one
            if (c0.color != 0) {
                const SolveCell t = c0;
                c0 = c1;
                c1 = t;
            }
            float* P = which ? V.py : V.px;
            const float h0 = which ? c0.hy : c0.hx, h1 = which ? c1.hy : c1.hx;
            float v0 = c0.mine ? P[c0.j] : 0.0f, v1 = c1.mine ? P[c1.j] : 0.0f;
#pragma unroll 1
            for (int s = 0; s < COARSE_SWEEPS; s++) {
                solveUpdate(P, c0, h0, v0);
                barSub(1 + which, npair);
                solveUpdate(P, c1, h1, v1);
                barSub(1 + which, npair);
            }
        }
        __syncthreads();
    }
#pragma unroll 1
    for (int l = (int)L - 1; l >= (int)lc; l--) {
        const SLv V = slv(sm, off, D, (uint32_t)l);
        const SLv U = slv(sm, off, D, (uint32_t)l + 1u);
        const int n = V.w * V.h;
#pragma unroll 1
        for (int j = tid; j < n; j += nt) {
            if (V.rho[j] <= 0.0f) continue;
            const int cy = slvRow(V, j);
            V2 e = prolongedFrom(U.rho, U.px, U.py, U.w, U.h, j - cy * V.w, cy);
            V.px[j] = V.px[j] + e.x;
            V.py[j] = V.py[j] + e.y;
        }
        __syncthreads();
        slv_smooth(V, (uint32_t)l, tid, nt);
    }
}

// A coarse level's cell as the reference's field holds it.
__device__ __forceinline__ void keepLevelCell(const Dev& D, uint32_t l, uint32_t j, float px, float py, float rx, float ry,
                                              float rho) {
    float4* f = reinterpret_cast<float4*>(D.field) + D.level_start[l] + 2u * j;
    f[0] = make_float4(px, py, rx, ry);
    f[1] = make_float4(rho, 0.0f, 0.0f, 0.0f);
}

// The levels lc (restricted already, in the scratch) down to the coarsest and
// back up to lc, in one CTA's shared memory: smoothRed/Black, restrictLevel,
// solve (40 SOR sweep pairs, omega 1.8), prolong (fluid.wgsl:2318-2470).
// Each level's face coefficients are worked out once, when its densities
// are in place, and read by its sweeps and by the restriction below it.
// Level lc's results go to its ux, uy; with KEEP, every level's words also
// to field's coarse levels, as the reference's passes leave them.
template <class T, bool KEEP = false>
__device__ void coarseLevels(const Dev& D, const FastW& F, const W& w, uint32_t lc, float* sm, uint32_t* off) {
    const uint32_t L = D.levels;
    const int tid = (int)threadIdx.x, nt = (int)blockDim.x;
    if (tid == 0) {
        uint32_t o = 0;
#pragma unroll 1
        for (uint32_t l = lc; l <= L; l++) {
            off[l] = o;
            o += SLV_ARRAYS * D.level_w[l] * D.level_h[l];
        }
    }
    __syncthreads();
    {
        const SLv V = slv(sm, off, D, lc);
        const LRef<T> G = lref<T>(F, lc);
        const int n = V.w * V.h;
#pragma unroll 1
        for (int j = tid; j < n; j += nt) {
            V.px[j] = ld(G.px + j);
            V.py[j] = ld(G.py + j);
            V.rx[j] = ld(G.rx + j);
            V.ry[j] = ld(G.ry + j);
            V.rho[j] = ld(G.rho + j);
        }
        __syncthreads();
    }
    coarseCore(D, w, lc, sm, off);
    {
        const SLv V = slv(sm, off, D, lc);
        auto* ox = upx<T>(F, lc);
        auto* oy = upy<T>(F, lc);
        const int n = V.w * V.h;
#pragma unroll 1
        for (int j = tid; j < n; j += nt) {
            st(ox + j, V.px[j]);
            st(oy + j, V.py[j]);
        }
    }
    if (KEEP) {
#pragma unroll 1
        for (uint32_t l = lc; l <= L; l++) {
            const SLv V = slv(sm, off, D, l);
            const int n = V.w * V.h;
            for (int j = tid; j < n; j += nt) keepLevelCell(D, l, (uint32_t)j, V.px[j], V.py[j], V.rx[j], V.ry[j], V.rho[j]);
        }
    }
}

template <bool ONE, class T>
__global__ void __launch_bounds__(1024) k_fCoarse(Batch Bt, const __grid_constant__ WorldSrc<ONE> src) {
    __shared__ WorldCopy wc_;
    if (!ONE) worldCopyInit(wc_);
    extern __shared__ float sm[];
    __shared__ uint32_t off[WIG_MG_LEVELS + 1];
    FOR_ITEMS(Bt, L_ONE, it) {
        FAST_ITEM(Bt, it, D, F, w, unused_);
        (void)unused_;
        if (D.st->cont == 0u) continue;
        coarseLevels<T>(D, F, w, F.lc, sm, off);
        __syncthreads();
    }
}

// ---------------------------------------------------------------- the coarse levels on a cluster
//
// A single world whose coarse kernel starts at a level of more than
// COARSE_CTA_CELLS cells (at 1024 x 1024: 128 x 128, with the coarse_cells
// knob at 16384) runs its coarse levels on one thread-block cluster of
// CLUSTER_CTAS CTAs instead of one CTA, in their distributed shared memory.
// Each level of more than RANK0_CELLS cells is cut into strips of rows, a
// strip a CTA, its nine arrays (px, py, rx, ry, rho, b0..b3) in that CTA's
// shared memory at the same offsets in every CTA; a neighbour's row across a
// strip's edge is read from the owning CTA (cluster.map_shared_rank).  The
// levels of at most RANK0_CELLS cells are CTA 0's alone (coarseCore, as in
// the one-CTA kernel).  Every pass is the one-CTA kernel's, cell for cell, in
// the same arithmetic and order (the cells of a colour are independent), and
// a cluster barrier ends each pass whose results another CTA reads.  The
// levels it takes over from the tile kernels (the restrict-only launch of
// its first level stays) would each have been a launch of one wave of a few
// CTAs.
constexpr int CLUSTER_CTAS = 8;
constexpr uint32_t RANK0_CELLS = 1024;

enum { A_PX = 0, A_PY, A_RX, A_RY, A_RHO, A_B0, A_B1, A_B2, A_B3 };

// n / d for any 32-bit n, with mul = floor((2^32 - 1) / d): the multiply-high
// is the quotient or one below it.
__device__ __forceinline__ uint32_t divq(uint32_t n, uint32_t d, uint32_t mul) {
    uint32_t q = __umulhi(n, mul);
    if (n - q * d >= d) q += 1u;
    return q;
}

// A level cut into strips: this CTA's rows r0 .. r1 - 1 of rpr a CTA; array
// k of a CTA's rows at base + k n (n = rpr w floats).
struct DLv {
    float* base;
    int n, w, h, rpr, r0, r1;
    uint32_t wmul, rmul;
    __device__ float* a(int k) const { return base + k * n; }
};
// The strip levels' shared memory: level lc's from sm, each next level's
// after the one above it.
__host__ __device__ inline size_t stripFloats(uint32_t w, uint32_t h) {
    return (size_t)SLV_ARRAYS * ((h + CLUSTER_CTAS - 1) / CLUSTER_CTAS) * w;
}
__device__ __forceinline__ DLv dlv(float* sm, const Dev& D, uint32_t lc, uint32_t l, unsigned me) {
    for (uint32_t k = lc; k < l; k++) sm += stripFloats(D.level_w[k], D.level_h[k]);
    DLv V;
    V.base = sm;
    V.w = (int)D.level_w[l];
    V.h = (int)D.level_h[l];
    V.rpr = (V.h + CLUSTER_CTAS - 1) / CLUSTER_CTAS;
    V.n = V.rpr * V.w;
    V.r0 = min((int)me * V.rpr, V.h);
    V.r1 = min(V.r0 + V.rpr, V.h);
    V.wmul = 0xffffffffu / (uint32_t)V.w;
    V.rmul = 0xffffffffu / (uint32_t)V.rpr;
    return V;
}
// Row y of a strip level (its array 0; array k at + k n), in whichever CTA
// holds it.
__device__ __forceinline__ float* dlRow(const DLv& V, int y, unsigned me) {
    const unsigned o = divq((uint32_t)y, (uint32_t)V.rpr, V.rmul);
    float* p = V.base + (y - (int)o * V.rpr) * V.w;
    return o == me ? p : cooperative_groups::this_cluster().map_shared_rank(p, o);
}
// This CTA's own cell j (of (r1 - r0) w): its coordinates.
__device__ __forceinline__ void dlCell(const DLv& V, int j, int* x, int* y) {
    const int q = (int)divq((uint32_t)j, (uint32_t)V.w, V.wmul);
    *x = j - q * V.w;
    *y = V.r0 + q;
}

// slv_stencil of a strip level's cell (x, y) in row r (its rows above and
// below from whichever CTAs hold them): the neighbours clamped onto the cell
// past the level's edge (nbr), each beta times its potential, in order.
__device__ __forceinline__ void dl_stencil(const DLv& V, const float* r, int x, int y, unsigned me, float* sx, float* sy,
                                           float* dg) {
    const float* u = y > 0 ? dlRow(V, y - 1, me) : r;
    const float* d = y < V.h - 1 ? dlRow(V, y + 1, me) : r;
    const int xl = x > 0 ? x - 1 : x, xr = x < V.w - 1 ? x + 1 : x;
    const int n = V.n;
    const float b0 = r[A_B0 * n + x], b1 = r[A_B1 * n + x], b2 = r[A_B2 * n + x], b3 = r[A_B3 * n + x];
    *sx = (((0.0f + b0 * r[xl]) + b1 * r[xr]) + b2 * u[x]) + b3 * d[x];
    *sy = (((0.0f + b0 * r[n + xl]) + b1 * r[n + xr]) + b2 * u[n + x]) + b3 * d[n + x];
    *dg = (((0.0f + b0) + b1) + b2) + b3;
}

// slv_coefficients over this CTA's strip.
__device__ void dl_coefficients(const DLv& V, unsigned me) {
    const int n = (V.r1 - V.r0) * V.w;
#pragma unroll 1
    for (int j = (int)threadIdx.x; j < n; j += (int)blockDim.x) {
        int x, y;
        dlCell(V, j, &x, &y);
        const float* own = V.a(A_RHO);
        const float rho = own[j];
        float b[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (rho > 0.0f) {
            const float* u = y > 0 ? dlRow(V, y - 1, me) + A_RHO * V.n : nullptr;
            const float* d = y < V.h - 1 ? dlRow(V, y + 1, me) + A_RHO * V.n : nullptr;
            const float rn[4] = {x > 0 ? own[j - 1] : 0.0f, x < V.w - 1 ? own[j + 1] : 0.0f, u ? u[x] : 0.0f,
                                 d ? d[x] : 0.0f};
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if (!nbrIn(x, y, V.w, V.h, q)) continue;
                if (rn[q] >= 0.0f) b[q] = faceBeta(rho, rn[q]);
            }
        }
        V.a(A_B0)[j] = b[0];
        V.a(A_B1)[j] = b[1];
        V.a(A_B2)[j] = b[2];
        V.a(A_B3)[j] = b[3];
    }
}

// slv_sweep of one colour over this CTA's strip: of its cells 2k and
// 2k + 1 exactly one has each colour, so pair k gives the cell.
__device__ void dl_sweep(const DLv& V, uint32_t l, int color, float omega, unsigned me) {
    const int n = (V.r1 - V.r0) * V.w, pairs = (n + 1) / 2;
    const float h2 = (float)(1u << (2u * l));
#pragma unroll 1
    for (int k = (int)threadIdx.x; k < pairs; k += (int)blockDim.x) {
        int j = 2 * k, x, y;
        dlCell(V, j, &x, &y);
        if (((x + y) & 1) != color) {
            j++;
            if (++x == V.w) {
                x = 0;
                y++;
            }
        }
        if (j >= n) continue;
        if (V.a(A_RHO)[j] <= 0.0f) continue;
        float* r = V.base + (j - x);
        float sx, sy, dg;
        dl_stencil(V, r, x, y, me, &sx, &sy, &dg);
        if (dg <= 0.0f) continue;
        float* px = V.a(A_PX);
        float* py = V.a(A_PY);
        px[j] = mixf(px[j], (sx - h2 * V.a(A_RX)[j]) / dg, omega);
        py[j] = mixf(py[j], (sy - h2 * V.a(A_RY)[j]) / dg, omega);
    }
}

// restrictLevel into coarse cell (cx, cy) of level l from strip level U
// (level l - 1), as coarseCore restricts: the stencil from U's stored
// coefficients.
__device__ __forceinline__ void dl_restricted(const Dev& D, const W& w, uint32_t l, const DLv& U, int cx, int cy, unsigned me,
                                              float* px, float* py, float* rx_o, float* ry_o, float* rho_o) {
    const int span = 1 << l;
    if (span <= BLOCK) {
        I2 b{cx * span / BLOCK, cy * span / BLOCK};
        if (w.inBlocks(b) && (D.blocks[w.stateSlot(w.blockIndex(b))] & ACTIVE) == 0u) {
            *px = 0.0f; *py = 0.0f; *rx_o = 0.0f; *ry_o = 0.0f; *rho_o = 0.0f;
            return;
        }
    }
    const float inv_h2u = 1.0f / (float)(1u << (2u * (l - 1u)));
    const int n = U.n;
    float fluid = 0.0f, sum = 0.0f, rx = 0.0f, ry = 0.0f;
    bool air = false;
    for (int q = 0; q < 4; q++) {
        const int kx = 2 * cx + (q & 1), ky = 2 * cy + (q >> 1);
        if (kx >= U.w || ky >= U.h) continue;
        const float* r = dlRow(U, ky, me);
        const float rho = r[A_RHO * n + kx];
        if (rho == 0.0f) air = true;
        else if (rho > 0.0f) {
            float sx, sy, dg;
            dl_stencil(U, r, kx, ky, me, &sx, &sy, &dg);
            fluid = fluid + 1.0f;
            sum = sum + rho;
            rx = rx + (r[A_RX * n + kx] - (sx - (dg + 0.0f) * r[kx]) * inv_h2u);
            ry = ry + (r[A_RY * n + kx] - (sy - (dg + 0.0f) * r[n + kx]) * inv_h2u);
        }
    }
    const float rho = air ? 0.0f : (fluid > 0.0f ? sum / fluid : -1.0f);
    *px = 0.0f;
    *py = 0.0f;
    *rx_o = rho > 0.0f ? rx * 0.25f : 0.0f;
    *ry_o = rho > 0.0f ? ry * 0.25f : 0.0f;
    *rho_o = rho;
}

// prolonged (fluid.wgsl:2478-2497) of fine cell (cx, cy) from strip level
// U: prolongedFrom's loads and weights, U's two rows from their CTAs.
__device__ __forceinline__ V2 dl_prolonged(const DLv& U, int cx, int cy, unsigned me) {
    const int kx = cx / 2, ky = cy / 2;
    const int sx = (cx & 1) == 1 ? 1 : -1, sy = (cy & 1) == 1 ? 1 : -1;
    const int ox[4] = {0, sx, 0, sx}, oy[4] = {0, 0, sy, sy};
    const float wt[4] = {9.0f, 3.0f, 3.0f, 1.0f};
    const bool row2 = ky + sy >= 0 && ky + sy < U.h;
    const float* r0 = dlRow(U, ky, me);
    const float* r1 = row2 ? dlRow(U, ky + sy, me) : r0;
    const int n = U.n;
    float rq[4], xq[4], yq[4];
    bool inq[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int ax_ = kx + ox[q], ay_ = ky + oy[q];
        inq[q] = !(ax_ < 0 || ay_ < 0 || ax_ >= U.w || ay_ >= U.h);
        const float* r = oy[q] == 0 ? r0 : r1;
        const int c = inq[q] ? ax_ : kx;
        rq[q] = r[A_RHO * n + c];
        xq[q] = r[c];
        yq[q] = r[n + c];
    }
    float ax = 0.0f, ay = 0.0f, weight = 0.0f;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        if (!inq[q]) continue;
        const float r = rq[q];
        if (r < 0.0f) continue;
        weight = weight + wt[q];
        if (r > 0.0f) {
            ax = ax + wt[q] * xq[q];
            ay = ay + wt[q] * yq[q];
        }
    }
    const float ww = fmaxf(weight, 1e-6f);
    return V2{ax / ww, ay / ww};
}

// The cluster's shared memory (floats a CTA) for a world from level lc: each
// strip level's rows of one CTA, then CTA 0's levels ls .. L; 0 when the
// coarsest level has more than RANK0_CELLS cells.
__host__ __device__ inline size_t clusterFloats(const uint32_t* lw, const uint32_t* lh, uint32_t lc, uint32_t L,
                                                uint32_t* ls_out) {
    size_t n = 0;
    uint32_t l = lc;
    for (; l <= L && lw[l] * lh[l] > RANK0_CELLS; l++) n += stripFloats(lw[l], lh[l]);
    if (ls_out) *ls_out = l;
    if (l > L) return 0;
    for (uint32_t k = l; k <= L; k++) n += (size_t)SLV_ARRAYS * lw[k] * lh[k];
    return n;
}

template <class T>
__global__ void __launch_bounds__(1024) k_fCoarseCluster(Batch Bt, const __grid_constant__ WorldSrc<true> src) {
    extern __shared__ float sm[];
    __shared__ uint32_t off[WIG_MG_LEVELS + 1];
    namespace cgs = cooperative_groups;
    cgs::cluster_group cl = cgs::this_cluster();
    const unsigned me = cl.block_rank();
    const World& Wd = src.w;
    const Dev& D = Wd.D;
    const FastW& F = Wd.S;
    const W w(D);
    (void)Bt;
    // every CTA reads the same word: all go on, or all return, together
    if (D.st->cont == 0u) return;
    const uint32_t lc = F.lc, L = D.levels;
    uint32_t ls = lc;
    clusterFloats(D.level_w, D.level_h, lc, L, &ls);
    // CTA 0's levels ls .. L after the strip levels lc .. ls - 1
    float* sm0 = sm;
    for (uint32_t l = lc; l < ls; l++) sm0 += stripFloats(D.level_w[l], D.level_h[l]);
    if (threadIdx.x == 0) {
        uint32_t o = 0;
        for (uint32_t l = ls; l <= L; l++) {
            off[l] = o;
            o += SLV_ARRAYS * D.level_w[l] * D.level_h[l];
        }
    }
    // level lc's rows from the scratch (restricted by the down kernel)
    {
        const DLv A = dlv(sm, D, lc, lc, me);
        const LRef<T> G = lref<T>(F, lc);
        const int n = (A.r1 - A.r0) * A.w;
#pragma unroll 1
        for (int j = (int)threadIdx.x; j < n; j += (int)blockDim.x) {
            const int g = A.r0 * A.w + j;
            A.a(A_PX)[j] = ld(G.px + g);
            A.a(A_PY)[j] = ld(G.py + g);
            A.a(A_RX)[j] = ld(G.rx + g);
            A.a(A_RY)[j] = ld(G.ry + g);
            A.a(A_RHO)[j] = ld(G.rho + g);
        }
    }
    cl.sync();
    // down the strip levels
    for (uint32_t l = lc; l < ls; l++) {
        const DLv A = dlv(sm, D, lc, l, me);
        if (l > lc) {
            const DLv U = dlv(sm, D, lc, l - 1u, me);
            const int n = (A.r1 - A.r0) * A.w;
#pragma unroll 1
            for (int j = (int)threadIdx.x; j < n; j += (int)blockDim.x) {
                int x, y;
                dlCell(A, j, &x, &y);
                dl_restricted(D, w, l, U, x, y, me, &A.a(A_PX)[j], &A.a(A_PY)[j], &A.a(A_RX)[j], &A.a(A_RY)[j],
                              &A.a(A_RHO)[j]);
            }
            cl.sync();
        }
        dl_coefficients(A, me);
        __syncthreads();
        dl_sweep(A, l, 0, SMOOTH_OMEGA, me);
        cl.sync();
        dl_sweep(A, l, 1, SMOOTH_OMEGA, me);
        cl.sync();
    }
    // CTA 0: level ls restricted from the last strip level, then the levels
    // below it and back up, in its own shared memory
    if (me == 0u) {
        const DLv U = dlv(sm, D, lc, ls - 1u, me);
        const SLv S = slv(sm0, off, D, ls);
        const int n = S.w * S.h;
#pragma unroll 1
        for (int j = (int)threadIdx.x; j < n; j += (int)blockDim.x) {
            const int cy = slvRow(S, j), cx = j - cy * S.w;
            dl_restricted(D, w, ls, U, cx, cy, me, &S.px[j], &S.py[j], &S.rx[j], &S.ry[j], &S.rho[j]);
        }
        __syncthreads();
        coarseCore(D, w, ls, sm0, off);
    }
    cl.sync();
    // up the strip levels: prolong from the level below (CTA 0's or a strip
    // level), then both colours
    for (int l = (int)ls - 1; l >= (int)lc; l--) {
        const DLv A = dlv(sm, D, lc, (uint32_t)l, me);
        const int n = (A.r1 - A.r0) * A.w;
        if (l + 1 == (int)ls) {
            // CTA 0's level ls, at offset 0 of its levels there
            const int lw = (int)D.level_w[ls], lh = (int)D.level_h[ls];
            const int nl = lw * lh;
            const float* b0 = cl.map_shared_rank(sm0, 0u);
#pragma unroll 1
            for (int j = (int)threadIdx.x; j < n; j += (int)blockDim.x) {
                if (A.a(A_RHO)[j] <= 0.0f) continue;
                int x, y;
                dlCell(A, j, &x, &y);
                const V2 e = prolongedFrom(b0 + 4 * nl, b0, b0 + nl, lw, lh, x, y);
                A.a(A_PX)[j] = A.a(A_PX)[j] + e.x;
                A.a(A_PY)[j] = A.a(A_PY)[j] + e.y;
            }
        } else {
            const DLv U = dlv(sm, D, lc, (uint32_t)l + 1u, me);
#pragma unroll 1
            for (int j = (int)threadIdx.x; j < n; j += (int)blockDim.x) {
                if (A.a(A_RHO)[j] <= 0.0f) continue;
                int x, y;
                dlCell(A, j, &x, &y);
                const V2 e = dl_prolonged(U, x, y, me);
                A.a(A_PX)[j] = A.a(A_PX)[j] + e.x;
                A.a(A_PY)[j] = A.a(A_PY)[j] + e.y;
            }
        }
        cl.sync();
        dl_sweep(A, (uint32_t)l, 0, SMOOTH_OMEGA, me);
        cl.sync();
        dl_sweep(A, (uint32_t)l, 1, SMOOTH_OMEGA, me);
        cl.sync();
    }
    // level lc's rows to its way-up potentials
    {
        const DLv A = dlv(sm, D, lc, lc, me);
        const int n = (A.r1 - A.r0) * A.w;
        auto* ox = upx<T>(F, lc);
        auto* oy = upy<T>(F, lc);
#pragma unroll 1
        for (int j = (int)threadIdx.x; j < n; j += (int)blockDim.x) {
            const int g = A.r0 * A.w + j;
            st(ox + g, A.a(A_PX)[j]);
            st(oy + g, A.a(A_PY)[j]);
        }
    }
}

// The CG kernels: a warp a tile of 8x8 cells, lane l the cells l and l + 32
// of the tile (rows l / 8 and l / 8 + 4), so a tile's tree of 64 (its first
// step adds l + 32 to l, the rest are shuffles) needs no barrier and no
// shared memory; a warp has two tiles' loads in flight.  A CTA takes a
// contiguous run of the active blocks, world by world, and counts each
// world's tiles once.  What bounds them is latency: per launch the chain
// state -> block index -> cells -> partial -> count -> the last CTA's sum
// of all the partials, against 2-5 us for their bytes on the 1024x1024
// world.  As four 64-thread tiles a 256-thread CTA under a barrier an item
// they took 15-18 us a launch there (83-95 us on the 2048x2048 column).
constexpr int CG_THREADS = 512, CG_WARPS = CG_THREADS / 32;

// The CTA's run over the active blocks, a world's part of it at a time:
// body(world, its active count, the part's first tile, its tiles).
template <bool ONE, class Body>
__device__ __forceinline__ void forTileRuns(const Batch& Bt, const WorldSrc<ONE>& src, WorldCopy& wc, Body body) {
    const uint32_t n = Bt.n(L_ACT), per = (n + gridDim.x - 1u) / gridDim.x;
    uint32_t g = blockIdx.x * per;
    const uint32_t e = min(g + per, n);
    while (g < e) {
        const uint32_t it = Bt.item(L_ACT, g), j0 = Bt.unit(it);
        const World& Wd = src.get(Bt, it, wc);
        const uint32_t na = W(Wd.D).activeCount();
        // (a world's items are its units 0 .. na - 1 in order)
        const uint32_t m = max(min(e - g, na - j0), 1u);
        body(Wd, na, j0, m);
        g += m;
    }
}

// prolongFine (fluid.wgsl:2500-2512) of cell c, and its rim for the
// relaxation after: the cell's words and the prolongation's loaded together,
// then used for a liquid cell only.  With KEEP the rim also goes where
// relaxRims leaves it (counters' G_RIM).  (A lane a quad of cells, whose
// nine coarse cells it loads once, was slower: 32 us a launch against 21 on
// a 48-world batch, for want of loads in flight.)
template <class T, bool KEEP = false>
__device__ __forceinline__ void prolongFineCell(const Dev& D, const FastW& F, const W& w, I2 c) {
    const uint32_t i = w.cellIndex(c);
    const uint32_t mk = F.Z.mask[i];
    const float2 p = F.Z.pot[i];
    const V2 e = prolongedFrom(lref<T>(F, 1u).rho, upx<T>(F, 1u), upy<T>(F, 1u), (int)D.level_w[1], (int)D.level_h[1], c.x, c.y);
    if ((mk & FM_LIQUID) == 0u) return;
    const float2 v = make_float2(p.x + e.x, p.y + e.y);
    F.Z.pot[i] = v;
    F.Z.rim[i] = v;
    if (KEEP) {
        *w.gwp(i, G_RIM) = __float_as_uint(v.x);
        *w.gwp(i, G_RIM + 1u) = __float_as_uint(v.y);
    }
}

template <bool ONE, class T>
__global__ void k_fProlongFine(Batch Bt, const __grid_constant__ WorldSrc<ONE> src) {
    __shared__ WorldCopy wc_;
    if (!ONE) worldCopyInit(wc_);
    FOR_ITEMS(Bt, L_ACT, it) {
        FAST_ITEM(Bt, it, D, F, w, wid);
        if (D.st->cont == 0u) continue;
        const I2 c = lidCell(w, wid);
        if (w.inWorld(c)) prolongFineCell<T>(D, F, w, c);
    }
}

// ================================================================ conjugate gradients

// A lane's two cells of tile wid: their indices and whether they are in the
// world (a ragged world's last blocks), and the tile's block.
struct TileLane {
    uint32_t n, i[2];
    int x, y[2];
    bool in[2];
};
__device__ __forceinline__ TileLane tileLane(const W& w, uint32_t wid, bool live) {
    TileLane t;
    const int lane = (int)(threadIdx.x & 31u);
    t.n = live ? w.D.blocks[w.activeSlot(wid)] : 0u;
    const I2 b = w.blockAt(t.n);
    t.x = b.x * BLOCK + (lane & 7);
#pragma unroll
    for (int h = 0; h < 2; h++) {
        t.y[h] = b.y * BLOCK + (lane >> 3) + 4 * h;
        t.in[h] = live && w.inWorld(I2{t.x, t.y[h]});
        t.i[h] = t.in[h] ? w.cellIndex(I2{t.x, t.y[h]}) : 0u;
    }
    return t;
}

template <class T, int NC, int NT>
__device__ __forceinline__ void sumBlocksCg(uint32_t B, const T* part, T* s, T (&out)[NC]) {
    sumColumns<T, NC, NT>(B, part, s);
    treeColumns<T, NC>(s);
#pragma unroll
    for (int c = 0; c < NC; c++) out[c] = s[256 * c];
}

// Counts the CTA's m tiles of a world whose partials its warps' first lanes
// have written; true in the CTA that counted the world's last tile (a
// threadfence reduction's test).  first(): thread 0's, before the count.
template <class First>
__device__ __forceinline__ bool countTiles(uint32_t* counter, uint32_t m, uint32_t total, First first) {
    __shared__ int last;
    if ((threadIdx.x & 31u) == 0u) __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        first();
        const uint32_t old = atomicAdd(counter, m);
        last = old + m == total ? 1 : 0;
        if (last) {
            *counter = 0u;
            __threadfence();
        }
    }
    __syncthreads();
    return last != 0;
}

// A world's partial sums as a kernel writes them: component c of block b at
// c * B + b, in FP64 or f32.
struct Parts {
    double* d;
    float* f;
};

// cgRho's sums (fluid.wgsl:2736-2750) of tiles j[0] and, when two, j[1].
__device__ __forceinline__ void rhoTiles(const Dev& D, const FastW& F, const W& w, const uint32_t (&j)[2], bool two, bool f64,
                                         const Parts& out) {
    const Fine& Z = F.Z;
    const uint32_t lane = threadIdx.x & 31u;
    TileLane t[2];
    uint32_t mk[2][2];
    float z[2][2], r[2][2], q[2][2];
#pragma unroll
    for (int u = 0; u < 2; u++) t[u] = tileLane(w, j[u], u == 0 || two);
#pragma unroll
    for (int u = 0; u < 2; u++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const uint32_t i = t[u].i[h];
            mk[u][h] = Z.mask[i];
            z[u][h] = Z.pot[i].x;
            r[u][h] = F.R[i];
            q[u][h] = F.Q[i];
        }
#pragma unroll
    for (int u = 0; u < 2; u++) {
        if (u == 1 && !two) break;  // (warp-uniform)
        const bool f0 = t[u].in[0] && (mk[u][0] & FM_LIQUID) != 0u, f1 = t[u].in[1] && (mk[u][1] & FM_LIQUID) != 0u;
        // the f32 trees only without FP64 dots, which read none of them
        if (f64) {
            const double x = warpTree(f0 ? (double)r[u][0] * (double)z[u][0] : 0.0, f1 ? (double)r[u][1] * (double)z[u][1] : 0.0);
            const double y = warpTree(f0 ? (double)q[u][0] * (double)z[u][0] : 0.0, f1 ? (double)q[u][1] * (double)z[u][1] : 0.0);
            if (lane == 0u) {
                out.d[t[u].n] = x;
                out.d[D.B + t[u].n] = y;
            }
        } else {
            const float x = warpTree(f0 ? r[u][0] * z[u][0] : 0.0f, f1 ? r[u][1] * z[u][1] : 0.0f);
            const float y = warpTree(f0 ? q[u][0] * z[u][0] : 0.0f, f1 ? q[u][1] * z[u][1] : 0.0f);
            if (lane == 0u) {
                out.f[t[u].n] = x;
                out.f[D.B + t[u].n] = y;
            }
        }
    }
}

// cgRho + cgBeta (fluid.wgsl:2736-2764).
template <bool ONE>
__global__ void __launch_bounds__(CG_THREADS, 2) k_fRhoBeta(Batch Bt, const __grid_constant__ WorldSrc<ONE> src) {
    __shared__ WorldCopy wc_;
    if (!ONE) worldCopyInit(wc_);
    __shared__ double s64[512];
    const uint32_t warp = threadIdx.x >> 5;
    forTileRuns<ONE>(Bt, src, wc_, [&](const World& Wd, uint32_t na, uint32_t j0, uint32_t m) {
        const Dev& D = Wd.D;
        const FastW& F = Wd.S;
        const W w(D);
        if (D.st->cont == 0u) return;
        const bool f64 = D.st->f64 != 0u;
        const uint32_t cycle = D.st->cycle;
#pragma unroll 1
        for (uint32_t t = warp; t < m; t += 2u * CG_WARPS) {
            const uint32_t j[2] = {j0 + t, j0 + t + CG_WARPS};
            rhoTiles(D, F, w, j, t + CG_WARPS < m, f64, Parts{F.part64, F.part32});
        }
        if (!countTiles(&D.st->fdone[1], m, na, [] {})) return;
        if (f64) {
            double v[2];
            sumBlocksCg<double, 2, CG_THREADS>(D.B, F.part64, s64, v);
            if (threadIdx.x == 0) {
                D.st->rz = v[0];
                D.st->beta = (cycle == 0u || D.st->pq <= 0.0) ? 0.0 : -v[1] / D.st->pq;
            }
        } else {
            float v[2];
            sumBlocksCg<float, 2, CG_THREADS>(D.B, F.part32, reinterpret_cast<float*>(s64), v);
            if (threadIdx.x == 0) {
                D.st->rz32 = v[0];
                D.st->beta32 = (cycle == 0u || D.st->pq32 <= 0.0f) ? 0.0f : -v[1] / D.st->pq32;
            }
        }
    });
}

// cgDirection + cgApply (fluid.wgsl:2767-2795) of tile j: the direction p =
// z + beta p_old of the tile's cells and of the 32 cells around it, a cell
// of these a lane (worked again from their z and p_old, the same
// arithmetic), in the warp's 10x10 of shared memory; q = A p, and the tile's
// tree of p q.  p_old is read from one of the two p arrays and p written
// to the other (by the iteration's parity), so no warp reads a p that
// another writes in the pass.
__device__ __forceinline__ void applyTile(const Dev& D, const FastW& F, const W& w, uint32_t j, bool odd, bool f64, float beta,
                                          double beta64, float* sp, const Parts& out) {
    const Fine& Z = F.Z;
    const float* Pold = odd ? F.P2 : F.P;
    float* Pnew = odd ? F.P : F.P2;
    const uint32_t lane = threadIdx.x & 31u;
    // the lane's cell around the tile: left and right columns, rows above
    // and below, 8 lanes each
    const int side = (int)(lane >> 3), at = (int)(lane & 7u);
    const int ox = side == 0 ? -1 : side == 1 ? BLOCK : at, oy = side == 2 ? -1 : side == 3 ? BLOCK : at;
    auto dir = [&](float z, float p) { return f64 ? (float)((double)z + beta64 * (double)p) : z + beta * p; };
    const TileLane t = tileLane(w, j, true);
    const I2 b = w.blockAt(t.n);
    const I2 oc{b.x * BLOCK + ox, b.y * BLOCK + oy};
    const bool oin = w.inWorld(oc);
    const uint32_t oi = oin ? w.cellIndex(oc) : 0u;
    const float oz = Z.pot[oi].x, op = Pold[oi];
    float4 bb[2];
    float z[2], po[2];
    uint32_t mk[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const uint32_t i = t.i[h];
        mk[h] = Z.mask[i];
        bb[h] = Z.b[i];
        z[h] = Z.pot[i].x;
        po[h] = Pold[i];
    }
    float p[2];
    const int c0 = ((int)(lane >> 3) + 1) * RIM + (int)(lane & 7u) + 1;
    sp[(oy + 1) * RIM + ox + 1] = dir(oz, op);
#pragma unroll
    for (int h = 0; h < 2; h++) {
        p[h] = dir(z[h], po[h]);
        sp[c0 + 4 * RIM * h] = p[h];
    }
    __syncwarp();
    float q[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int c = c0 + 4 * RIM * h;
        q[h] = 0.0f;
        if (t.in[h] && (mk[h] & FM_LIQUID) != 0u) {
            float sum = 0.0f;
            if (mk[h] & 1u) sum = sum + bb[h].x * sp[c - 1];
            if (mk[h] & 2u) sum = sum + bb[h].y * sp[c + 1];
            if (mk[h] & 4u) sum = sum + bb[h].z * sp[c - RIM];
            if (mk[h] & 8u) sum = sum + bb[h].w * sp[c + RIM];
            const float dgp = diagOf(bb[h]) + ((mk[h] & FM_PIN) != 0u ? PIN : 0.0f);
            q[h] = dgp * p[h] - sum + 0.0f;
        } else {
            p[h] = 0.0f;
        }
        if (t.in[h]) {
            Pnew[t.i[h]] = p[h];
            F.Q[t.i[h]] = q[h];
        }
    }
    if (f64) {
        const double x = warpTree((double)p[0] * (double)q[0], (double)p[1] * (double)q[1]);
        if (lane == 0u) out.d[t.n] = x;
    } else {
        const float x = warpTree(p[0] * q[0], p[1] * q[1]);
        if (lane == 0u) out.f[t.n] = x;
    }
    __syncwarp();  // the warp's p is free for its next tile
}

// With free bodies A p needs every body's J p first: cgDirection and
// cgBodyP (fluid.wgsl:2767-2776, :2828-2836) of tile j.
__device__ __forceinline__ void directionTile(const Dev& D, const FastW& F, const W& w, uint32_t j, uint32_t cycle, bool f64,
                                              float beta, double beta64) {
    const bool odd = (cycle & 1u) != 0u;
    const float* Pold = odd ? F.P2 : F.P;
    float* Pnew = odd ? F.P : F.P2;
    const TileLane t = tileLane(w, j, true);
#pragma unroll
    for (int h = 0; h < 2; h++) {
        if (!t.in[h]) continue;
        const uint32_t i = t.i[h], mk = F.Z.mask[i];
        const float z = F.Z.pot[i].x, po = Pold[i];
        float p = 0.0f;
        if ((mk & FM_LIQUID) != 0u) p = f64 ? (float)((double)z + beta64 * (double)po) : z + beta * po;
        Pnew[i] = p;
        if ((mk & FM_BODY) != 0u) addPressurePush(w, I2{t.x, t.y[h]}, p, PUSH_P0 + cycle % 2u);
    }
}
// ... and cgApply (fluid.wgsl:2779-2795) of tile j from them, its f32 sums
// also where the reference's cg keeps them.
__device__ __forceinline__ void applyCoupledTile(const Dev& D, const FastW& F, const W& w, uint32_t j, uint32_t cycle,
                                                 bool f64, const Parts& out) {
    const float* P = (cycle & 1u) != 0u ? F.P : F.P2;
    const TileLane t = tileLane(w, j, true);
    float p[2] = {0.0f, 0.0f}, q[2] = {0.0f, 0.0f};
#pragma unroll
    for (int h = 0; h < 2; h++) {
        if (!t.in[h]) continue;
        const uint32_t i = t.i[h], mk = F.Z.mask[i];
        if ((mk & FM_LIQUID) != 0u) {
            const float4 bb = F.Z.b[i];
            const float b[4] = {bb.x, bb.y, bb.z, bb.w};
            p[h] = P[i];
            float sum = 0.0f;
#pragma unroll
            for (int d = 0; d < 4; d++)
                if (mk & (1u << d)) sum = sum + b[d] * P[nbr(i, t.x, t.y[h], D.W, D.H, d)];
            const float dgp = diagOf(bb) + ((mk & FM_PIN) != 0u ? PIN : 0.0f);
            q[h] = dgp * p[h] - sum + ((mk & FM_BODY) != 0u ? couplingAt(w, I2{t.x, t.y[h]}, PUSH_P0 + cycle % 2u) : 0.0f);
        }
        F.Q[i] = q[h];
    }
    const float x32 = warpTree(p[0] * q[0], p[1] * q[1]);
    const double x = warpTree((double)p[0] * (double)q[0], (double)p[1] * (double)q[1]);
    if ((threadIdx.x & 31u) == 0u) {
        if (f64) out.d[t.n] = x;
        else out.f[t.n] = x32;
        reinterpret_cast<float4*>(D.cg)[D.C + t.n] = make_float4(x32, 0.0f, 0.0f, 0.0f);
    }
}

// cgDirection + cgApply + cgAlpha (fluid.wgsl:2767-2814).
template <bool ONE>
__global__ void __launch_bounds__(CG_THREADS, 2) k_fApplyAlpha(Batch Bt, const __grid_constant__ WorldSrc<ONE> src) {
    __shared__ WorldCopy wc_;
    if (!ONE) worldCopyInit(wc_);
    __shared__ double s64[256];
    __shared__ float tp[CG_WARPS][RIM * RIM];
    const uint32_t warp = threadIdx.x >> 5;
    forTileRuns<ONE>(Bt, src, wc_, [&](const World& Wd, uint32_t na, uint32_t j0, uint32_t m) {
        const Dev& D = Wd.D;
        const FastW& F = Wd.S;
        const W w(D);
        if (D.st->cont == 0u) return;
        const bool f64 = D.st->f64 != 0u, odd = (D.st->cycle & 1u) != 0u;
        const float beta = D.st->beta32;
        const double beta64 = D.st->beta;
#pragma unroll 1
        for (uint32_t t = warp; t < m; t += CG_WARPS)
            applyTile(D, F, w, j0 + t, odd, f64, beta, beta64, tp[warp], Parts{F.pq64, F.pq32});
        if (!countTiles(&D.st->fdone[2], m, na, [] {})) return;
        if (f64) {
            double v[1];
            sumBlocksCg<double, 1, CG_THREADS>(D.B, F.pq64, s64, v);
            if (threadIdx.x == 0) {
                D.st->pq = v[0];
                D.st->alpha = v[0] <= 0.0 ? 0.0 : D.st->rz / v[0];
            }
        } else {
            float v[1];
            sumBlocksCg<float, 1, CG_THREADS>(D.B, F.pq32, reinterpret_cast<float*>(s64), v);
            if (threadIdx.x == 0) {
                D.st->pq32 = v[0];
                D.st->alpha32 = v[0] <= 0.0f ? 0.0f : D.st->rz32 / v[0];
            }
        }
    });
}

// cgUpdate's work (fluid.wgsl:2857-2880) on tiles j[0] and, when two, j[1],
// with each tile's sum of r^2 when tol; the lane's largest |r| (bits of a
// non-negative float).
__device__ __forceinline__ uint32_t updateTiles(const Dev& D, const FastW& F, const W& w, const uint32_t (&j)[2], bool two,
                                                const float* P, bool f64, bool tol, float alpha, double alpha64) {
    const Fine& Z = F.Z;
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t most = 0u;
    TileLane t[2];
    uint32_t mk[2][2];
    float vx[2][2], vy[2][2], vz[2][2], vw[2][2], py[2][2];
#pragma unroll
    for (int u = 0; u < 2; u++) t[u] = tileLane(w, j[u], u == 0 || two);
#pragma unroll
    for (int u = 0; u < 2; u++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const uint32_t i = t[u].i[h];
            mk[u][h] = Z.mask[i];
            vx[u][h] = F.X[i];
            vy[u][h] = F.R[i];
            vz[u][h] = P[i];
            vw[u][h] = F.Q[i];
            py[u][h] = Z.pot[i].y;
        }
#pragma unroll
    for (int u = 0; u < 2; u++) {
        if (u == 1 && !two) break;  // (warp-uniform)
        double r2[2] = {0.0, 0.0};
#pragma unroll
        for (int h = 0; h < 2; h++) {
            if (!t[u].in[h] || (mk[u][h] & FM_LIQUID) == 0u) continue;
            const uint32_t i = t[u].i[h];
            float r, x;
            if (f64) {
                r = (float)((double)vy[u][h] - alpha64 * (double)vw[u][h]);
                x = (float)((double)vx[u][h] + alpha64 * (double)vz[u][h]);
            } else {
                r = vy[u][h] - alpha * vw[u][h];
                x = vx[u][h] + alpha * vz[u][h];
            }
            F.X[i] = x;
            F.R[i] = r;
            Z.pot[i].x = 0.0f;
            Z.rim[i] = make_float2(0.0f, py[u][h]);
            most = max(most, __float_as_uint(fabsf(r)));
            r2[h] = (double)r * (double)r;
        }
        if (tol) {
            const double v = warpTree(r2[0], r2[1]);
            if (lane == 0u) D.norm64[t[u].n] = v;
        }
    }
    return most;
}

// cgUpdate (fluid.wgsl:2852-2880), the tolerance form's norm, and the loop's
// condition: a world iterates again unless its solve has converged
// (converged, fluid.wgsl:2223-2226) or max_cycles are done; the loop runs on
// while any world does.
template <bool ONE>
__global__ void __launch_bounds__(CG_THREADS, 2) k_fUpdate(Batch Bt, const __grid_constant__ WorldSrc<ONE> src) {
    __shared__ WorldCopy wc_;
    if (!ONE) worldCopyInit(wc_);
    __shared__ uint32_t runMost;  // the largest |r| of the current world's run (bits of a non-negative float)
    __shared__ double s64[256];
    if (threadIdx.x == 0) runMost = 0u;
    __syncthreads();
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    forTileRuns<ONE>(Bt, src, wc_, [&](const World& Wd, uint32_t na, uint32_t j0, uint32_t m) {
        const Dev& D = Wd.D;
        const FastW& F = Wd.S;
        const W w(D);
        if (D.st->cont == 0u) return;
        const uint32_t cycle = D.st->cycle;
        const bool f64 = D.st->f64 != 0u, tol = D.st->tol_mode != 0u;
        const float alpha = D.st->alpha32;
        const double alpha64 = D.st->alpha;
        const float* P = (cycle & 1u) ? F.P : F.P2;
        uint32_t most = 0u;
#pragma unroll 1
        for (uint32_t t = warp; t < m; t += 2u * CG_WARPS) {
            const uint32_t j[2] = {j0 + t, j0 + t + CG_WARPS};
            most = max(most, updateTiles(D, F, w, j, t + CG_WARPS < m, P, f64, tol, alpha, alpha64));
        }
        // the run's largest |r| into the world's residual slot (a max of
        // maxima: the same word), before its tiles are counted
        most = __reduce_max_sync(0xffffffffu, most);
        if (lane == 0u && most) atomicMax(&runMost, most);
        if (!countTiles(&D.st->fdone[3], m, na, [&] {
                atomicMax(&D.blocks[w.countSlot(COUNT_RESIDUAL + cycle % 3u)], runMost);
                runMost = 0u;
                __threadfence();
            }))
            return;
        double rr[1] = {0.0};
        if (tol) sumBlocksCg<double, 1, CG_THREADS>(D.B, D.norm64, s64, rr);
        if (threadIdx.x == 0) {
            bool conv;
            if (tol) {
                const double rel = D.st->bnorm2 > 0.0 ? sqrt(rr[0] / D.st->bnorm2) : 0.0;
                D.st->rel = rel;
                conv = rel <= D.st->tol;
            } else {
                conv = __uint_as_float(__ldcg(&D.blocks[w.countSlot(COUNT_RESIDUAL + cycle % 3u)])) < LIQUID_TOLERANCE;
            }
            const uint32_t next = cycle + 1u;
            // the mixed form checks the true residual every 8th iteration
            // and before it stops (k_fTrueCheck may then go on)
            const bool check = Bt.mixed != 0u && tol && (conv || (next % 8u) == 0u || next >= Bt.max_cycles);
            const uint32_t cont = (!conv && next < Bt.max_cycles) ? 1u : 0u;
            D.st->cycle = next;
            D.st->cont = cont;
            D.st->check = check ? 1u : 0u;
            if (check && Bt.cond_check) cudaGraphSetConditional(Bt.cond_check, 1u);
            if (cont) {
                *Bt.loop = 1u;
                if (Bt.cond) cudaGraphSetConditional(Bt.cond, 1u);
            }
        }
    });
}

// The true residual -(b + A x) of liquid cell i at c, worked in FP64 from the
// FP32 solution, and (floor2) the square of the FP32 rounding of A x there:
// u (|d x| + sum |beta x_n|), u = 2^-24 (the CG's own residual cannot stay
// below that floor's norm).
__device__ __forceinline__ double trueResidualAt(const Dev& D, const FastW& F, I2 c, uint32_t i, double* floor2) {
    const Fine& Z = F.Z;
    const uint32_t m = Z.mask[i];
    const float4 b4 = Z.b[i];
    const float bb[4] = {b4.x, b4.y, b4.z, b4.w};
    const double dx = (double)(diagOf(b4) + ((m & FM_PIN) != 0u ? PIN : 0.0f)) * (double)F.X[i];
    double ax = dx, mag = fabs(dx);
#pragma unroll
    for (int d = 0; d < 4; d++)
        if (m & (1u << d)) {
            const double t = (double)bb[d] * (double)F.X[nbr(i, c.x, c.y, D.W, D.H, d)];
            ax = ax - t;
            mag = mag + fabs(t);
        }
    const double f = mag * 5.9604644775390625e-8;
    *floor2 = f * f;
    return -((double)D.field[8u * (size_t)i + 1u] + ax);
}

// A tile's sums of the squares of its cells' true residuals and floors, of
// block b at b and B + b of out.
__device__ __forceinline__ void trueCheckTile(const Dev& D, const FastW& F, const W& w, uint32_t j, double* out) {
    const TileLane t = tileLane(w, j, true);
    double r2[2] = {0.0, 0.0}, f2[2] = {0.0, 0.0};
#pragma unroll
    for (int h = 0; h < 2; h++)
        if (t.in[h] && (F.Z.mask[t.i[h]] & FM_LIQUID) != 0u) {
            const double r = trueResidualAt(D, F, I2{t.x, t.y[h]}, t.i[h], &f2[h]);
            r2[h] = r * r;
        }
    const double t2 = warpTree(r2[0], r2[1]), u2 = warpTree(f2[0], f2[1]);
    if ((threadIdx.x & 31u) == 0u) {
        out[t.n] = t2;
        out[D.B + t.n] = u2;
    }
}
// The true residual's norm and the floor's, relative to b's; and whether the
// true one has drifted above twice the recursive one plus four floors (the
// low-precision preconditioner's rounding lost the recursion's accuracy).
__device__ __forceinline__ void trueRel(double rr, double ff, double bn, double* rel, double* flo) {
    *rel = bn > 0.0 ? sqrt(rr / bn) : 0.0;
    *flo = bn > 0.0 ? sqrt(ff / bn) : 0.0;
}
__device__ __forceinline__ bool drifted(double rel_true, double rel, double flo) { return rel_true > 2.0 * rel + 4.0 * flo; }
// The true residual put in for the recursive one.
__device__ __forceinline__ void trueFixTile(const Dev& D, const FastW& F, const W& w, uint32_t j) {
    const TileLane t = tileLane(w, j, true);
#pragma unroll
    for (int h = 0; h < 2; h++)
        if (t.in[h] && (F.Z.mask[t.i[h]] & FM_LIQUID) != 0u) {
            double f2;
            F.R[t.i[h]] = (float)trueResidualAt(D, F, I2{t.x, t.y[h]}, t.i[h], &f2);
        }
}

// The mixed form's guard, over the worlds k_fUpdate flagged: a world whose
// true residual has drifted goes on with it put in (k_fTrueFix), else it
// stops or goes on as k_fUpdate decided.
template <bool ONE>
__global__ void __launch_bounds__(CG_THREADS, 2) k_fTrueCheck(Batch Bt, const __grid_constant__ WorldSrc<ONE> src) {
    __shared__ WorldCopy wc_;
    if (!ONE) worldCopyInit(wc_);
    __shared__ double s64[512];
    forTileRuns<ONE>(Bt, src, wc_, [&](const World& Wd, uint32_t na, uint32_t j0, uint32_t m) {
        const Dev& D = Wd.D;
        const W w(D);
        if (D.st->check == 0u) return;
#pragma unroll 1
        for (uint32_t t = threadIdx.x >> 5; t < m; t += CG_WARPS) trueCheckTile(D, Wd.S, w, j0 + t, Wd.S.part64);
        if (!countTiles(&D.st->fdone[4], m, na, [] {})) return;
        double v[2];
        sumBlocksCg<double, 2, CG_THREADS>(D.B, Wd.S.part64, s64, v);
        if (threadIdx.x == 0) {
            double rel, flo;
            trueRel(v[0], v[1], D.st->bnorm2, &rel, &flo);
            D.st->rel_true = rel;
            D.st->check = 0u;
            if (drifted(rel, D.st->rel, flo)) {
                D.st->drift = 1u;
                if (Bt.cond_drift) cudaGraphSetConditional(Bt.cond_drift, 1u);
                const uint32_t cont = D.st->cycle < Bt.max_cycles ? 1u : 0u;
                D.st->cont = cont;
                if (cont) {
                    *Bt.loop = 1u;
                    if (Bt.cond) cudaGraphSetConditional(Bt.cond, 1u);
                }
            }
        }
    });
}

// The worlds k_fTrueCheck found drifted.
template <bool ONE>
__global__ void __launch_bounds__(CG_THREADS, 2) k_fTrueFix(Batch Bt, const __grid_constant__ WorldSrc<ONE> src) {
    __shared__ WorldCopy wc_;
    if (!ONE) worldCopyInit(wc_);
    forTileRuns<ONE>(Bt, src, wc_, [&](const World& Wd, uint32_t na, uint32_t j0, uint32_t m) {
        const W w(Wd.D);
        if (Wd.D.st->drift == 0u) return;
#pragma unroll 1
        for (uint32_t t = threadIdx.x >> 5; t < m; t += CG_WARPS) trueFixTile(Wd.D, Wd.S, w, j0 + t);
    });
}

// An iteration's start: the loop stops unless a world's k_fUpdate says
// otherwise; each world still iterating (all of them on the first
// iteration) clears its next residual slot and counts the iteration
// (cgUpdate's first lines, fluid.wgsl:2852-2856), and one with no block
// worked on stops there, as cgUpdate's converged test stops it.
__global__ void k_fLoopStart(Batch Bt) {
    if (threadIdx.x != 0) return;
    if (blockIdx.x == 0) {
        *Bt.loop = 0u;
        if (Bt.cond) cudaGraphSetConditional(Bt.cond, 0u);
        if (Bt.cond_check) cudaGraphSetConditional(Bt.cond_check, 0u);
        if (Bt.cond_drift) cudaGraphSetConditional(Bt.cond_drift, 0u);
    }
    FOR_ITEMS(Bt, L_ONE, it) {
        ITEM_WORLD(Bt, it, D, w, unused_);
        (void)unused_;
        StepState* st = D.st;
        st->drift = 0u;
        if (st->cycle == 0u) st->cont = 1u;
        if (st->cont == 0u) continue;
        const uint32_t cycle = st->cycle;
        D.blocks[w.countSlot(COUNT_RESIDUAL + (cycle + 1u) % 3u)] = 0u;
        D.blocks[w.countSlot(COUNT_CYCLES)] += 1u;
        if (w.activeCount() == 0u) {
            st->cycle = cycle + 1u;
            st->cont = 0u;
        }
    }
}

// cgFinish (fluid.wgsl:2884-2893) and the solve's values back into the
// reference's buffers: field's pressure, divergence left (-r) and drift
// potential, cg's (x, r, p, Ap); and the residual slots the converged
// iterations the reference still dispatches would clear (cgUpdate's first
// lines run whether or not the iteration is skipped).
template <bool ONE>
__global__ void k_fFinish(Batch Bt, const __grid_constant__ WorldSrc<ONE> src) {
    __shared__ WorldCopy wc_;
    if (!ONE) worldCopyInit(wc_);
    if (threadIdx.x == 0) {
        FOR_ITEMS(Bt, L_ONE, ot) {
            ITEM_WORLD(Bt, ot, D, w, unused_);
            (void)unused_;
            for (uint32_t c = D.st->cycle; c < Bt.max_cycles; c++)
                D.blocks[w.countSlot(COUNT_RESIDUAL + (c + 1u) % 3u)] = 0u;
        }
    }
    FOR_ITEMS(Bt, L_ACT, it) {
        FAST_ITEM(Bt, it, D, F, w, wid);
        const Fine& Z = F.Z;
        I2 c = lidCell(w, wid);
        if (!w.inWorld(c)) continue;
        uint32_t i = w.cellIndex(c);
        float* f = w.fv(2u * i);
        f[0] = F.X[i];
        if ((Z.mask[i] & FM_LIQUID) != 0u) f[1] = -F.R[i];
        w.fv(2u * i + 1u)[0] = Z.pot[i].y;
        // the last iteration's p: P2 after an odd number of iterations
        const float* P = (D.st->cycle & 1u) ? F.P2 : F.P;
        reinterpret_cast<float4*>(D.cg)[i] = make_float4(F.X[i], F.R[i], P[i], F.Q[i]);
        *w.gwp(i, G_REGION) = 0u;
    }
}


// ================================================================ one world's solve in one launch
//
// All the iterations of a single world's solve in one kernel, by a group of
// CTAs: each pass of an iteration is a phase, every warp (or half CTA)
// taking its share of the phase's tiles, the phases separated by the
// group's barrier; the coarse levels are CTA 0's, in its shared memory.
// Same tiles, same values, same order of every sum as the passes' kernels.
//
// Why: an iteration is 14 to 16 launches, each of which costs about 2.5 us
// between kernels in the step's graph and starts by loading what the last
// one knew (its world's state, its list's length): on small worlds most of
// the solve, on a 1024x1024 world 50 of its 185 us an iteration.  A barrier
// among the CTAs of a cluster is under 1 us, among those of a grid about
// 1.5 us.
constexpr int SOLVE_THREADS = 1024, SOLVE_WARPS = SOLVE_THREADS / 32, TEAM = SOLVE_THREADS / 2;

// The CTAs of one cluster.
struct ClusterGroup {
    static constexpr bool EAGER = true;  // (downTile)
    uint32_t rank, n;
    __device__ explicit ClusterGroup(StepState*)
        : rank(cooperative_groups::this_cluster().block_rank()), n(cooperative_groups::this_cluster().num_blocks()) {}
    __device__ __forceinline__ bool sync() {
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
        return true;
    }
};

// The CTAs of a cooperative launch (all resident): arrivals counted up in
// the world's StepState, the k-th barrier passed at k n of them.  Each wait
// is bounded: past g_spin_limit polls a CTA records ERR_BARRIER and marks the
// count as given up (wig_wait.h), and every CTA returns false from here on.
struct GridGroup {
    static constexpr bool EAGER = false;
    StepState* st;
    uint32_t rank, n, target;
    __device__ explicit GridGroup(StepState* s) : st(s), rank(blockIdx.x), n(gridDim.x), target(0u) {}
    __device__ bool sync() {
        __shared__ int s_ok;
        target += n;
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t v, it = 0;
            const uint32_t limit = g_spin_limit;
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&st->bar_count) : "memory");
            while (true) {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&st->bar_count) : "memory");
                if (barrierOver(v, target)) break;
                if (++it > limit) {
                    atomicOr(&st->err, ERR_BARRIER);
                    v = atomicOr(&st->bar_count, BARRIER_GAVE_UP) | BARRIER_GAVE_UP;
                    break;
                }
            }
            s_ok = barrierGaveUp(v) ? 0 : 1;
        }
        __syncthreads();
        return s_ok != 0;
    }
};

// A world of more blocks has its block sums' columns shared by the group's
// CTAs (a warp a column) and a barrier more; below, every CTA sums them all
// itself (a round of loads for 4096 blocks, about 1 us).
constexpr uint32_t SPLIT_BLOCKS = 8192;
static_assert(SPLIT_BLOCKS >= COMPACT_BLOCKS && COL64_VALUES >= 2u * 256u, "a splitting world has its columns' memory");

// sumBlocks of NC components of the partials, for every CTA of the group
// (all its threads): the sums in s[256 c].  col: 512 values of scratch.
template <class T, int NC, class Group>
__device__ __forceinline__ bool groupSums(Group& g, uint32_t B, const T* part, T* s, float* sm, double* col64) {
    if (B <= SPLIT_BLOCKS) {
        sumColumns<T, NC, SOLVE_THREADS>(B, part, s);
        treeColumns<T, NC>(s);
        return true;
    }
    T* col = reinterpret_cast<T*>(col64);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t id = g.rank + g.n * warp;
    if (id < 256u * NC) {
        constexpr uint32_t ROWS = 256u;
        T* rows = reinterpret_cast<T*>(sm) + ROWS * warp;
        const T* at = part + (size_t)B * (id >> 8);
        const uint32_t li = id & 255u;
        T acc = T(0);
        for (uint32_t r0 = 0; r0 * 256u < B; r0 += ROWS) {
            T v[ROWS / 32u];
#pragma unroll
            for (uint32_t u = 0; u < ROWS / 32u; u++) {
                const uint32_t k = (r0 + lane + 32u * u) * 256u + li;
                v[u] = k < B ? __ldcg(at + k) : T(0);
            }
            __syncwarp();
#pragma unroll
            for (uint32_t u = 0; u < ROWS / 32u; u++) rows[lane + 32u * u] = v[u];
            __syncwarp();
            if (lane == 0u) {
                const uint32_t m = min(ROWS, (B + 255u) / 256u - r0);  // (the rest are +0)
#pragma unroll 8
                for (uint32_t k = 0; k < m; k++) acc = acc + rows[k];
            }
        }
        if (lane == 0u) col[id] = acc;
    }
    if (!g.sync()) return false;
    for (uint32_t k = threadIdx.x; k < 256u * NC; k += SOLVE_THREADS) s[k] = __ldcg(col + k);
    treeColumns<T, NC>(s);
    return true;
}

// The columns' warps must be there: 32 a CTA, so 16 CTAs of a group that
// splits.
constexpr uint32_t SPLIT_CTAS = 16;

// BODIES: the world's free bodies coupled in (A = L + J^T M^-1 J: cgBodyP's
// phase more an iteration), and the solve's scratch words left in the
// reference's buffers too.
template <class Group, class T, bool BODIES>
__global__ void __launch_bounds__(SOLVE_THREADS, 1) k_fSolve(const __grid_constant__ World Wd, uint32_t max_cycles) {
    extern __shared__ __align__(16) float sm[];
    __shared__ double s64[512];
    __shared__ uint32_t s_off[WIG_MG_LEVELS + 1];
    __shared__ uint32_t s_most;
    const Dev& D = Wd.D;
    const FastW& F = Wd.S;
    const W w(D);
    StepState* st = D.st;
    Group g(st);
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const bool f64 = st->f64 != 0u, tol = st->tol_mode != 0u;
    const double tolerance = st->tol, bnorm2 = st->bnorm2;
    const uint32_t shift_first = st->shift_first & 1u;
    const uint32_t na = w.activeCount(), lc = F.lc;
    float* s32 = reinterpret_cast<float*>(s64);
    // the group's first warp of a phase over tiles, and its stride
    const uint32_t w0 = g.rank * SOLVE_WARPS + warp, wn = g.n * SOLVE_WARPS;
    const Team<TEAM> tm{(int)(tid % TEAM), 2 + (int)(tid / TEAM)};
    LevelTile& lt = reinterpret_cast<LevelTile*>(sm)[tid / TEAM];
    const uint32_t t0 = g.rank + g.n * (tid / TEAM), tn = 2u * g.n;
    if (tid == 0u) s_most = 0u;
    double rz = 0.0, pq = 0.0, rel = 1.0, rel_true = 0.0;
    float rz32 = 0.0f, pq32 = 0.0f;
    uint32_t cycle = 0;
    if (na == 0u) {
        // nothing to solve: the first iteration counted, as cgUpdate counts it
        if (g.rank == 0u && tid == 0u) {
            D.blocks[w.countSlot(COUNT_RESIDUAL + 1u)] = 0u;
            D.blocks[w.countSlot(COUNT_CYCLES)] += 1u;
            st->cycle = 1u;
            st->cont = 0u;
        }
        return;
    }
    for (bool more = true; more;) {
        if (g.rank == 0u && tid == 0u) {
            // cgUpdate's first lines: the next slot cleared, the iteration counted
            D.blocks[w.countSlot(COUNT_RESIDUAL + (cycle + 1u) % 3u)] = 0u;
            D.blocks[w.countSlot(COUNT_CYCLES)] += 1u;
        }
        float2* rim = reinterpret_cast<float2*>(sm) + RIM * RXS * warp;
#pragma unroll 1
        for (uint32_t half = 0; half < 2u; half++) {
            // relax: the active blocks' tiles, and on the shifted tiling the edge tiles
            const int shift = (shift_first ^ half) ? BLOCK / 2 : 0;
            const uint32_t total = na + (shift ? D.edge_tiles : 0u);
#pragma unroll 1
            for (uint32_t j = w0; j < total; j += wn) relaxTile<T>(D, F, w, na, j, shift, rim);
            if (!g.sync()) return;
            if (half) break;
#pragma unroll 1
            for (uint32_t l = 1; l <= lc; l++) {
                const uint32_t tiles = levelTiles(D.level_w[l], D.level_h[l]);
#pragma unroll 1
                for (uint32_t t = t0; t < tiles; t += tn) {
                    if (l == 1u) downTile<T, TEAM, true, false, Group::EAGER || BODIES>(D, F, w, l, t, cycle == 0u, lt, tm);
                    else downTile<T, TEAM, false, false, Group::EAGER || BODIES>(D, F, w, l, t, cycle == 0u, lt, tm);
                }
                if (!g.sync()) return;
            }
            if (g.rank == 0u) coarseLevels<T, BODIES>(D, F, w, lc, sm, s_off);
            if (!g.sync()) return;
#pragma unroll 1
            for (uint32_t l = lc - 1u; l >= 1u; l--) {
                const uint32_t tiles = levelTiles(D.level_w[l], D.level_h[l]);
#pragma unroll 1
                for (uint32_t t = t0; t < tiles; t += tn) upTile<T, TEAM, Group::EAGER || BODIES>(D, F, l, t, lt, tm);
                if (!g.sync()) return;
            }
#pragma unroll 1
            for (uint32_t j = w0; j < na; j += wn) {
                const I2 b = w.activeBlock(j);
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const I2 c{b.x * BLOCK + (int)(lane & 7u), b.y * BLOCK + (int)(lane >> 3) + 4 * h};
                    if (w.inWorld(c)) prolongFineCell<T, BODIES>(D, F, w, c);
                }
            }
            if (!g.sync()) return;
        }
        // cgRho, cgBeta
        double beta = 0.0, alpha = 0.0;
        float beta32 = 0.0f, alpha32 = 0.0f;
#pragma unroll 1
        for (uint32_t j0 = w0; j0 < na; j0 += 2u * wn) {
            const uint32_t j[2] = {j0, j0 + wn};
            rhoTiles(D, F, w, j, j0 + wn < na, f64, Parts{F.part64, F.part32});
        }
        if (!g.sync()) return;
        if (f64) {
            if (!groupSums<double, 2>(g, D.B, F.part64, s64, sm, F.col64)) return;
            rz = s64[0];
            beta = (cycle == 0u || pq <= 0.0) ? 0.0 : -s64[256] / pq;
        } else {
            if (!groupSums<float, 2>(g, D.B, F.part32, s32, sm, F.col64)) return;
            rz32 = s32[0];
            beta32 = (cycle == 0u || pq32 <= 0.0f) ? 0.0f : -s32[256] / pq32;
        }
        __syncthreads();  // the sums are read: their memory is free
        // cgDirection, cgApply, cgAlpha
        const bool odd = (cycle & 1u) != 0u;
        if (BODIES) {
#pragma unroll 1
            for (uint32_t j = w0; j < na; j += wn) directionTile(D, F, w, j, cycle, f64, beta32, beta);
            if (!g.sync()) return;
#pragma unroll 1
            for (uint32_t j = w0; j < na; j += wn) applyCoupledTile(D, F, w, j, cycle, f64, Parts{F.pq64, F.pq32});
        } else {
#pragma unroll 1
            for (uint32_t j = w0; j < na; j += wn)
                applyTile(D, F, w, j, odd, f64, beta32, beta, sm + RIM * RIM * warp, Parts{F.pq64, F.pq32});
        }
        if (!g.sync()) return;
        if (f64) {
            if (!groupSums<double, 1>(g, D.B, F.pq64, s64, sm, F.col64)) return;
            pq = s64[0];
            alpha = pq <= 0.0 ? 0.0 : rz / pq;
        } else {
            if (!groupSums<float, 1>(g, D.B, F.pq32, s32, sm, F.col64)) return;
            pq32 = s32[0];
            alpha32 = pq32 <= 0.0f ? 0.0f : rz32 / pq32;
        }
        __syncthreads();
        if (BODIES && g.rank == 0u) {
            // the bodies' sums of this iteration's direction, done with,
            // emptied for the iteration after next (fluid.wgsl:2808-2813),
            // and the scalars where the reference's cg keeps them
            const uint32_t which = PUSH_P0 + cycle % 2u;
            for (uint32_t k = tid; k < MAX_BODIES * 6u; k += SOLVE_THREADS) D.pushes[pushSlot(k / 6u, which, 0u) + k % 6u] = 0u;
            if (tid == 0u)
                reinterpret_cast<float4*>(D.cg)[D.C + D.B] =
                    f64 ? make_float4((float)rz, (float)alpha, (float)beta, (float)pq) : make_float4(rz32, alpha32, beta32, pq32);
        }
        // cgUpdate
        uint32_t most = 0u;
#pragma unroll 1
        for (uint32_t j0 = w0; j0 < na; j0 += 2u * wn) {
            const uint32_t j[2] = {j0, j0 + wn};
            most = max(most, updateTiles(D, F, w, j, j0 + wn < na, odd ? F.P : F.P2, f64, tol, alpha32, alpha));
        }
        most = __reduce_max_sync(0xffffffffu, most);
        if (lane == 0u && most) atomicMax(&s_most, most);
        __syncthreads();
        if (tid == 0u) {
            if (s_most) atomicMax(&D.blocks[w.countSlot(COUNT_RESIDUAL + cycle % 3u)], s_most);
            s_most = 0u;
        }
        if (!g.sync()) return;
        // converged (fluid.wgsl:2223-2226) for the next iteration: every CTA
        // decides the same from the same sums
        bool conv;
        if (tol) {
            if (!groupSums<double, 1>(g, D.B, D.norm64, s64, sm, F.col64)) return;
            rel = bnorm2 > 0.0 ? sqrt(s64[0] / bnorm2) : 0.0;
            conv = rel <= tolerance;
        } else {
            conv = __uint_as_float(__ldcg(&D.blocks[w.countSlot(COUNT_RESIDUAL + cycle % 3u)])) < LIQUID_TOLERANCE;
        }
        __syncthreads();
        cycle++;
        more = !conv && cycle < max_cycles;
        if (sizeof(T) == 2 && (conv || cycle % 8u == 0u || cycle >= max_cycles)) {
            // the mixed form's guard (k_fTrueCheck, k_fTrueFix)
#pragma unroll 1
            for (uint32_t j = w0; j < na; j += wn) trueCheckTile(D, F, w, j, F.part64);
            if (!g.sync()) return;
            if (!groupSums<double, 2>(g, D.B, F.part64, s64, sm, F.col64)) return;
            double flo;
            trueRel(s64[0], s64[256], bnorm2, &rel_true, &flo);
            __syncthreads();
            if (drifted(rel_true, rel, flo)) {
                more = cycle < max_cycles;
#pragma unroll 1
                for (uint32_t j = w0; j < na; j += wn) trueFixTile(D, F, w, j);
                if (!g.sync()) return;
            }
        }
    }
    if (BODIES) {
        // the levels above the coarse ones (no CTA writes them any more)
        for (uint32_t l = 1; l < lc; l++) {
            const LRef<T> V = lref<T>(F, l);
            const auto* ux = upx<T>(F, l);
            const auto* uy = upy<T>(F, l);
            const uint32_t n = D.level_w[l] * D.level_h[l];
            for (uint32_t j = g.rank * SOLVE_THREADS + tid; j < n; j += g.n * SOLVE_THREADS) {
                const float rho = ld(V.rho + j);
                const float2 h = V.rhs(j);
                keepLevelCell(D, l, j, rho > 0.0f ? ld(ux + j) : 0.0f, rho > 0.0f ? ld(uy + j) : 0.0f, h.x, h.y, rho);
            }
        }
    }
    if (g.rank == 0u && tid == 0u) {
        st->cycle = cycle;
        st->cont = 0u;
        st->rel = rel;
        st->rel_true = rel_true;
    }
}

}  // namespace

size_t fast_coarse_smem(const Dev& D, uint32_t lc) {
    size_t n = 0;
    for (uint32_t l = lc; l <= D.levels; l++) n += (size_t)D.level_w[l] * D.level_h[l];
    return SLV_ARRAYS * n * sizeof(float);
}

size_t fast_cluster_smem(const Dev& D, uint32_t lc) {
    if (lc < 1u || lc > D.levels || (size_t)D.level_w[lc] * D.level_h[lc] <= COARSE_CTA_CELLS) return 0;
    return clusterFloats(D.level_w, D.level_h, lc, D.levels, nullptr) * sizeof(float);
}

void fast_zero_level0(const World& Wd, cudaStream_t s) { k_fZero<<<148 * 4, 256, 0, s>>>(Wd.D, Wd.S); }

void fast_zero_idle(const Batch& Bt, const BatchShape& S, cudaStream_t s) {
    k_fZeroIdle<<<list_grid(S, L_WB, 32), 64, 0, s>>>(Bt);
}

// Launches kernel K's instance for the batch: the single-world one with
// the world as a parameter when `one` is given, else the table one.
#define LAUNCH(K, grid, block, smem, ...)                                                      \
    do {                                                                                       \
        if (one) K<true><<<(grid), (block), (smem), s>>>(Bt, WorldSrc<true>{*one}, ##__VA_ARGS__); \
        else K<false><<<(grid), (block), (smem), s>>>(Bt, WorldSrc<false>{}, ##__VA_ARGS__);       \
    } while (0)
// The same for a kernel over levels stored as T with N threads a CTA.
#define LAUNCH_TN(K, T, N, grid, smem, ...)                                                            \
    do {                                                                                               \
        if (one) K<true, T, N><<<(grid), (N), (smem), s>>>(Bt, WorldSrc<true>{*one}, ##__VA_ARGS__);    \
        else K<false, T, N><<<(grid), (N), (smem), s>>>(Bt, WorldSrc<false>{}, ##__VA_ARGS__);          \
    } while (0)
// The down kernel with N threads a CTA, from level 0 (FINE) or a coarse level.
#define LAUNCH_DOWN(T, N, FINE, grid, l)                                                      \
    do {                                                                                      \
        if (one) k_fDown<true, T, N, FINE><<<(grid), (N), 0, s>>>(Bt, WorldSrc<true>{*one}, l); \
        else k_fDown<false, T, N, FINE><<<(grid), (N), 0, s>>>(Bt, WorldSrc<false>{}, l);       \
    } while (0)
// The same for a kernel over levels stored as T.
#define LAUNCH_T(K, T, grid, block, smem, ...)                                                        \
    do {                                                                                              \
        if (one) K<true, T><<<(grid), (block), (smem), s>>>(Bt, WorldSrc<true>{*one}, ##__VA_ARGS__);   \
        else K<false, T><<<(grid), (block), (smem), s>>>(Bt, WorldSrc<false>{}, ##__VA_ARGS__);         \
    } while (0)

void fast_setup(const Batch& Bt, const BatchShape& S, const World* one, cudaStream_t s, const Marker* m) {
    if (m) m->fn(m->ctx, WIG_SLOT_F_SETUP, 0);
    const unsigned grid = list_grid(S, L_ACT4, 8);
    if (one && one->D.motion) k_fSetup<true, true><<<grid, 256, 0, s>>>(Bt, WorldSrc<true>{*one});
    else if (one) k_fSetup<true, false><<<grid, 256, 0, s>>>(Bt, WorldSrc<true>{*one});
    else k_fSetup<false, false><<<grid, 256, 0, s>>>(Bt, WorldSrc<false>{});
    if (m) m->fn(m->ctx, WIG_SLOT_F_SETUP, 1);
}

// An IF node at the capture point of stream `outer`, on condition `h`; its
// body captured from `body` (launches on the given stream).
template <class Body>
cudaError_t captureIf(cudaStream_t outer, cudaGraphConditionalHandle h, cudaStream_t inner, Body body) {
    cudaStreamCaptureStatus cs;
    cudaGraph_t g = nullptr;
    const cudaGraphNode_t* deps = nullptr;
    size_t nd = 0;
    cudaError_t e = cudaStreamGetCaptureInfo(outer, &cs, nullptr, &g, &deps, &nd);
    if (e != cudaSuccess) return e;
    cudaGraphNodeParams cp = {};
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = h;
    cp.conditional.type = cudaGraphCondTypeIf;
    cp.conditional.size = 1;
    cudaGraphNode_t node;
    e = cudaGraphAddNode(&node, g, deps, nd, &cp);
    if (e != cudaSuccess) return e;
    e = cudaStreamUpdateCaptureDependencies(outer, &node, 1, cudaStreamSetCaptureDependencies);
    if (e != cudaSuccess) return e;
    e = cudaStreamBeginCaptureToGraph(inner, cp.conditional.phGraph_out[0], nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed);
    if (e != cudaSuccess) return e;
    body(inner);
    cudaGraph_t captured = nullptr;
    const cudaError_t e2 = cudaStreamEndCapture(inner, &captured);
    e = cudaGetLastError();
    return e != cudaSuccess ? e : e2;
}

template <class T>
uint32_t fast_cycle_t(const Batch& Bt0, const BatchShape& S, const World* one, cudaStream_t s, const Marker* m,
                      NestCapture* nest) {
    // the mixed form's check and fix: under IF nodes when captured, with
    // their conditions' handles in the kernels' Batch from the iteration's
    // start (k_fLoopStart clears them, k_fUpdate and k_fTrueCheck set them)
    Batch Bt = Bt0;
    cudaGraphConditionalHandle hc = 0, hd = 0;
    if (Bt.mixed && nest && nest->err == cudaSuccess) {
        cudaStreamCaptureStatus cs;
        cudaGraph_t g = nullptr;
        nest->err = cudaStreamGetCaptureInfo(s, &cs, nullptr, &g, nullptr, nullptr);
        if (nest->err == cudaSuccess) nest->err = cudaGraphConditionalHandleCreate(&hc, g, 0, cudaGraphCondAssignDefault);
        if (nest->err == cudaSuccess) nest->err = cudaGraphConditionalHandleCreate(&hd, g, 0, cudaGraphCondAssignDefault);
        Bt.cond_check = (unsigned long long)hc;
        Bt.cond_drift = (unsigned long long)hd;
    }
    // the CG kernels: at most a tile a warp
    const unsigned GC = std::max(std::min((S.max_items[L_ACT] + CG_WARPS - 1u) / CG_WARPS, 148u * S.cg_per_sm), 1u);
    const unsigned GR = std::max(std::min((S.max_items[L_RELAX] + 3u) / 4u, 148u * S.relax_per_sm), 1u);
    uint32_t launches = 0;
    auto mark = [&](int slot, int phase) {
        if (m) m->fn(m->ctx, slot, phase);
        if (phase) launches++;
    };
    mark(WIG_SLOT_F_LOOP, 0);
    k_fLoopStart<<<list_grid(S, L_ONE, 1), 32, 0, s>>>(Bt);
    mark(WIG_SLOT_F_LOOP, 1);
    mark(WIG_SLOT_F_RELAX, 0);
    LAUNCH_T(k_fRelax, T, GR, 128, 0, 0);
    mark(WIG_SLOT_F_RELAX, 1);
    // down: each world restricts its levels 1..lc by themselves and smooths
    // those above lc (a kernel a level), then its levels from lc are the
    // coarse kernel's; up: each level above lc prolonged and smoothed
    // a single world's levels of at most two tiles a multiprocessor: 512
    // threads a tile, so each thread takes fewer of its cells in turn
    auto wide = [&](uint32_t list) { return one != nullptr && S.max_items[list] <= 2u * 148u; };
    for (uint32_t l = 1; l <= S.lc_max; l++) {
        mark(WIG_SLOT_F_RESTRICT, 0);
        const uint32_t list = L_RES + l - 1u;
        const unsigned grid = list_grid(S, list, S.level_per_sm);
        if (l == 1u) {
            if (wide(list)) LAUNCH_DOWN(T, 512, true, grid, l);
            else LAUNCH_DOWN(T, 256, true, grid, l);
        } else {
            if (wide(list)) LAUNCH_DOWN(T, 512, false, grid, l);
            else LAUNCH_DOWN(T, 256, false, grid, l);
        }
        mark(WIG_SLOT_F_RESTRICT, 1);
    }
    mark(WIG_SLOT_F_COARSE, 0);
    if (S.cluster && one) {
        // one cluster of CLUSTER_CTAS CTAs
        cudaLaunchConfig_t c = {};
        c.gridDim = dim3(CLUSTER_CTAS);
        c.blockDim = dim3(1024);
        c.dynamicSmemBytes = S.coarse_smem;
        c.stream = s;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = CLUSTER_CTAS;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        c.attrs = at;
        c.numAttrs = 1;
        (void)cudaLaunchKernelEx(&c, k_fCoarseCluster<T>, Bt, WorldSrc<true>{*one});
    } else {
        LAUNCH_T(k_fCoarse, T, list_grid(S, L_ONE, 1), 1024, S.coarse_smem);
    }
    mark(WIG_SLOT_F_COARSE, 1);
    for (uint32_t l = S.lc_max; l >= 1; l--) {
        if (S.max_items[L_SM + l - 1u] == 0u) continue;
        mark(WIG_SLOT_F_PROLONG, 0);
        const uint32_t list = L_SM + l - 1u;
        if (wide(list))
            LAUNCH_TN(k_fUp, T, 512, list_grid(S, list, S.level_per_sm), 0, l);
        else
            LAUNCH_T(k_fUp, T, list_grid(S, list, S.level_per_sm), 256, 0, l);
        mark(WIG_SLOT_F_PROLONG, 1);
    }
    mark(WIG_SLOT_F_PROLONG_FINE, 0);
    LAUNCH_T(k_fProlongFine, T, list_grid(S, L_ACT, 32), 64, 0);
    mark(WIG_SLOT_F_PROLONG_FINE, 1);
    mark(WIG_SLOT_F_RELAX, 0);
    LAUNCH_T(k_fRelax, T, GR, 128, 0, 1);
    mark(WIG_SLOT_F_RELAX, 1);
    mark(WIG_SLOT_F_RHO_BETA, 0);
    LAUNCH(k_fRhoBeta, GC, CG_THREADS, 0);
    mark(WIG_SLOT_F_RHO_BETA, 1);
    mark(WIG_SLOT_F_APPLY_ALPHA, 0);
    LAUNCH(k_fApplyAlpha, GC, CG_THREADS, 0);
    mark(WIG_SLOT_F_APPLY_ALPHA, 1);
    mark(WIG_SLOT_F_UPDATE, 0);
    LAUNCH(k_fUpdate, GC, CG_THREADS, 0);
    mark(WIG_SLOT_F_UPDATE, 1);
    if (Bt.mixed && hc && hd) {
        // captured: launched only on the iterations that check (not counted
        // among every iteration's launches)
        if (nest->err == cudaSuccess)
            nest->err = captureIf(s, hc, nest->s, [&](cudaStream_t s) { LAUNCH(k_fTrueCheck, GC, CG_THREADS, 0); });
        if (nest->err == cudaSuccess)
            nest->err = captureIf(s, hd, nest->s, [&](cudaStream_t s) { LAUNCH(k_fTrueFix, GC, CG_THREADS, 0); });
    } else if (Bt.mixed) {
        mark(WIG_SLOT_F_UPDATE, 0);
        LAUNCH(k_fTrueCheck, GC, CG_THREADS, 0);
        mark(WIG_SLOT_F_UPDATE, 1);
        mark(WIG_SLOT_F_UPDATE, 0);
        LAUNCH(k_fTrueFix, GC, CG_THREADS, 0);
        mark(WIG_SLOT_F_UPDATE, 1);
    }
    return launches;
}

uint32_t fast_cycle(const Batch& Bt, const BatchShape& S, const World* one, cudaStream_t s, const Marker* m,
                    NestCapture* nest) {
    return Bt.mixed ? fast_cycle_t<__half>(Bt, S, one, s, m, nest) : fast_cycle_t<float>(Bt, S, one, s, m, nest);
}

void fast_finish(const Batch& Bt, const BatchShape& S, const World* one, cudaStream_t s, const Marker* m) {
    if (m) m->fn(m->ctx, WIG_SLOT_F_FINISH, 0);
    LAUNCH(k_fFinish, list_grid(S, L_ACT, 32), 64, 0);
    if (m) m->fn(m->ctx, WIG_SLOT_F_FINISH, 1);
}

cudaError_t fast_prepare_attributes() {
    // the limit is the kernel's, not a batch's (another batch's launches
    // come under it too): room for any
    const int b = (int)SOLVE_SMEM_MOST;
    cudaError_t e = cudaFuncSetAttribute(k_fCoarse<true, float>, cudaFuncAttributeMaxDynamicSharedMemorySize, b);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_fCoarse<false, float>, cudaFuncAttributeMaxDynamicSharedMemorySize, b);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_fCoarse<true, __half>, cudaFuncAttributeMaxDynamicSharedMemorySize, b);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_fCoarse<false, __half>, cudaFuncAttributeMaxDynamicSharedMemorySize, b);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_fCoarseCluster<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, b);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_fCoarseCluster<__half>, cudaFuncAttributeMaxDynamicSharedMemorySize, b);
    return e;
}

// A solve's shared memory from level lc: the coarse levels', and at least
// what the other phases take.
size_t solve_smem(const Dev& D, uint32_t lc) {
    const size_t least = std::max({2u * sizeof(LevelTile), (size_t)SOLVE_WARPS * RIM * RXS * sizeof(float2),
                                   (size_t)SOLVE_WARPS * 256u * sizeof(double)});
    return std::max(fast_coarse_smem(D, lc), least);
}

template <class Group, class T, bool BODIES>
cudaError_t solve_attributes(size_t smem, bool cluster) {
    cudaError_t e = cudaFuncSetAttribute(k_fSolve<Group, T, BODIES>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess && cluster)
        e = cudaFuncSetAttribute(k_fSolve<Group, T, BODIES>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return e;
}

// Launches k_fSolve<Group, T, BODIES> on n CTAs: one cluster, or a cooperative grid.
template <class Group, class T, bool BODIES>
cudaError_t solve_launch(const World& Wd, uint32_t max_cycles, uint32_t n, bool cluster, cudaStream_t s) {
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(n);
    c.blockDim = dim3(SOLVE_THREADS);
    c.dynamicSmemBytes = solve_smem(Wd.D, Wd.S.lc);
    c.stream = s;
    cudaLaunchAttribute at[1];
    if (cluster) {
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = n;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
    } else {
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
    }
    c.attrs = at;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, k_fSolve<Group, T, BODIES>, Wd, max_cycles);
}

cudaError_t fast_solve_shape(const Dev& D, SolveShape* out) {
    int dev = 0, sms = 0, per = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // the attributes are the kernels', not this world's: room for any
    const size_t most = SOLVE_SMEM_MOST;
    if (e == cudaSuccess) e = solve_attributes<GridGroup, float, false>(most, false);
    if (e == cudaSuccess) e = solve_attributes<GridGroup, float, true>(most, false);
    if (e == cudaSuccess) e = solve_attributes<GridGroup, __half, false>(most, false);
    if (e == cudaSuccess) e = solve_attributes<ClusterGroup, float, false>(most, true);
    if (e == cudaSuccess) e = solve_attributes<ClusterGroup, float, true>(most, true);
    if (e == cudaSuccess) e = solve_attributes<ClusterGroup, __half, false>(most, true);
    // the first level of at most COARSE_CTA_CELLS cells that fits a CTA with
    // the levels below it (a level a cell or two high only halves, so that
    // 4096 x 1 cells are 7680 with those below, 276 KB)
    out->lc = coarse_level(D, COARSE_CTA_CELLS);
    while (out->lc < D.levels && solve_smem(D, out->lc) > most) out->lc++;
    const size_t smem = solve_smem(D, out->lc);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_fSolve<GridGroup, float, true>, SOLVE_THREADS, smem);
    if (e != cudaSuccess) return e;
    if (per < 1) return cudaErrorInvalidConfiguration;
    out->grid = std::min((uint32_t)sms, std::max(SPLIT_CTAS, (D.B + GRID_TILES - 1u) / GRID_TILES));
    // the cluster, for a world of few blocks: the most CTAs that fit
    out->cluster = 0;
    if (D.B <= CLUSTER_BLOCKS) {
        for (uint32_t n = SOLVE_CLUSTER; n >= 4u && out->cluster == 0u; n /= 2u) {
            cudaLaunchConfig_t c = {};
            c.gridDim = dim3(n);
            c.blockDim = dim3(SOLVE_THREADS);
            c.dynamicSmemBytes = smem;
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = n;
            at[0].val.clusterDim.y = 1;
            at[0].val.clusterDim.z = 1;
            c.attrs = at;
            c.numAttrs = 1;
            int fit = 0;
            if (cudaOccupancyMaxActiveClusters(&fit, k_fSolve<ClusterGroup, float, true>, &c) == cudaSuccess && fit > 0) out->cluster = n;
            else cudaGetLastError();
        }
    }
    return cudaSuccess;
}

cudaError_t fast_solve(const Batch& Bt, const World& W0, const SolveShape& h, bool grid, cudaStream_t s, const Marker* m) {
    World Wd = W0;
    // (a coarse level of the cluster coarse kernel's is too large for one CTA)
    Wd.S.lc = std::max(Wd.S.lc, h.lc);
    if (m) m->fn(m->ctx, WIG_SLOT_F_SOLVE, 0);
    cudaError_t e;
    const bool bodies = Wd.D.motion != nullptr;
    if (!grid && h.cluster) {
        e = bodies      ? solve_launch<ClusterGroup, float, true>(Wd, Bt.max_cycles, h.cluster, true, s)
            : Bt.mixed  ? solve_launch<ClusterGroup, __half, false>(Wd, Bt.max_cycles, h.cluster, true, s)
                        : solve_launch<ClusterGroup, float, false>(Wd, Bt.max_cycles, h.cluster, true, s);
    } else {
        e = bodies      ? solve_launch<GridGroup, float, true>(Wd, Bt.max_cycles, h.grid, false, s)
            : Bt.mixed  ? solve_launch<GridGroup, __half, false>(Wd, Bt.max_cycles, h.grid, false, s)
                        : solve_launch<GridGroup, float, false>(Wd, Bt.max_cycles, h.grid, false, s);
    }
    if (m) m->fn(m->ctx, WIG_SLOT_F_SOLVE, 1);
    return e;
}

}  // namespace wig
