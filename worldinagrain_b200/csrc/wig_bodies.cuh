// wig_bodies.cuh — the free bodies' table and push sums as the passes and the
// solve read and add to them.
#pragma once
#include "wig_device.cuh"

namespace wig {

// ================================================================ free bodies
// (fluid.wgsl:1181-1470; the body table's words, js/shared.js:294-333).  The
// pushes are exact two-word sums (common.wgsl:1378-1412) added by atomics, so
// their totals do not depend on the order the cells add them in.

constexpr uint32_t MAX_BODIES = WIG_MAX_BODIES;
constexpr uint32_t PUSH_P0 = 0, PUSH_X = 2, PUSH_F = 3, PUSH_SURFACE = 4, PUSH_DRAG = 5;
constexpr float EXACT_COARSE = 16777216.0f;
struct V3 { float x, y, z; };

__device__ __forceinline__ uint32_t bodyWord(const W& w, uint32_t b, uint32_t k) {
    return w.D.motion[MAX_BODIES + b * WIG_BODY_TABLE_WORDS + k];
}
__device__ __forceinline__ float bodyF(const W& w, uint32_t b, uint32_t k) { return __uint_as_float(bodyWord(w, b, k)); }
__device__ __forceinline__ V2 bodyV(const W& w, uint32_t b, uint32_t k) { return V2{bodyF(w, b, k), bodyF(w, b, k + 1u)}; }
__device__ __forceinline__ uint32_t liquidSlot(uint32_t b, uint32_t k) { return WIG_BODY_LIQUID_BASE + b * WIG_BODY_LIQUID_WORDS + k; }
__device__ __forceinline__ bool bodyInSolve(const W& w, uint32_t b) {
    uint32_t flags = bodyWord(w, b, WIG_BW_FLAGS);
    return !((flags & WIG_BF_ALIVE) == 0u || (flags & WIG_BF_NEW) != 0u || bodyF(w, b, WIG_BW_MASS) <= 0.0f);
}
// rigidBodyOf (fluid.wgsl:1233-1248)
__device__ inline uint32_t rigidBodyOf(const W& w, uint4 v) {
    const uint32_t t = wordType(v.x);
    const wig_elem& e = w.elem(t);
    if (!wordHas(v.x, WIG_FL_LOOSE) || e.kind != WIG_KIND_SOLID || e.break_to == WIG_NO_ELEM) return NONE;
    const float id = f16_value(v.w & 0xffffu);
    if (id < 0.0f || id >= (float)MAX_BODIES) return NONE;
    const uint32_t b = f2u(id);
    return bodyInSolve(w, b) ? b : NONE;
}
__device__ __forceinline__ float rigidMass(const W& w, uint32_t b) { return bodyF(w, b, WIG_BW_MASS) + bodyF(w, b, WIG_BW_CARGO); }
__device__ __forceinline__ float rigidInertia(const W& w, uint32_t b) {
    return bodyF(w, b, WIG_BW_INERTIA) + bodyF(w, b, WIG_BW_CARGO_INERTIA);
}
__device__ __forceinline__ float bodyDensity(const W& w, uint32_t b) {
    return rigidMass(w, b) / fmaxf((float)bodyWord(w, b, WIG_BW_CELLS), 1.0f);
}
__device__ __forceinline__ bool isHeld(const W& w, uint32_t b) { return (bodyWord(w, b, WIG_BW_FLAGS) & WIG_BF_HELD) != 0u; }
// wetRegionAt (fluid.wgsl:592-595)
__device__ inline bool wetRegionAt(const W& w, uint4 v) {
    if (!w.D.motion) return false;
    const uint32_t b = rigidBodyOf(w, v);
    return b != NONE && (bodyWord(w, b, WIG_BW_FLAGS) & (WIG_BF_WET | WIG_BF_HELD)) == (WIG_BF_WET | WIG_BF_HELD);
}
// bodySweptSlot, claimStep (common.wgsl:316-385): cell i's stamp of step frame
__device__ __forceinline__ uint32_t claimStep(uint32_t frame) { return frame % WIG_CLAIM_PERIOD + 1u; }
__device__ __forceinline__ uint32_t bodySweptSlot(const W& w, uint32_t i, uint32_t frame) {
    const uint32_t tiles = (((uint32_t)w.D.W + WIG_BODY_TILE - 1u) / WIG_BODY_TILE) *
                           (((uint32_t)w.D.H + WIG_BODY_TILE - 1u) / WIG_BODY_TILE);
    const uint32_t base = 4u * tiles + WIG_BODY_STAT_WORDS + WIG_BODY_COUNTERS + MAX_BODIES + (2u + WIG_BODY_SUM_WORDS) * w.D.C;
    return base + 1u + tiles + 2u * w.D.C + w.D.C + 2u * i + (frame & 1u);
}
// cupOf, seamOf (fluid.wgsl:1252-1288): the body whose cup (seam) cell i was
// stamped last step, alive and weighed; cupBefore (fluid.wgsl:3521-3528):
// whose cup it was the step before, whatever the body's state now
__device__ inline uint32_t sweptBody(const W& w, uint32_t i, uint32_t frame, uint32_t seam) {
    if (!w.D.stamps || !w.D.motion) return NONE;
    const uint32_t key = w.D.stamps[bodySweptSlot(w, i, frame)];
    if ((key >> 12u) != claimStep(frame) || (key & 1u) != seam) return NONE;
    const uint32_t b = 2047u - ((key >> 1u) & 0x7ffu);
    return b < MAX_BODIES ? b : NONE;
}
__device__ inline uint32_t cupOf(const W& w, uint32_t i) {
    const uint32_t b = sweptBody(w, i, w.D.st->P.frame - 1u, 0u);
    return b != NONE && bodyInSolve(w, b) ? b : NONE;
}
__device__ inline uint32_t seamOf(const W& w, uint32_t i) {
    const uint32_t b = sweptBody(w, i, w.D.st->P.frame - 1u, 1u);
    return b != NONE && bodyInSolve(w, b) ? b : NONE;
}
__device__ __forceinline__ uint32_t cupBefore(const W& w, uint32_t i) { return sweptBody(w, i, w.D.st->P.frame - 2u, 0u); }
// rigidAt, heldAt (fluid.wgsl:1422-1458): the body classify put in the drift's z
__device__ inline uint32_t rigidAt(const W& w, I2 c) {
    if (!w.D.motion || !w.inWorld(c)) return NONE;
    const float z = w.fv(2u * w.cellIndex(c) + 1u)[2];
    const uint32_t b = f2u(fmaxf(-z, 1.0f)) - 1u;
    return (z < 0.0f && b < MAX_BODIES) ? b : NONE;
}
__device__ inline uint32_t heldAt(const W& w, I2 c) {
    if (!w.D.motion || !w.inWorld(c)) return NONE;
    const float z = w.fv(2u * w.cellIndex(c) + 1u)[2];
    const uint32_t b = f2u(fmaxf(-z, 1.0f)) - 1u;
    // (a slot past the table, from a drift word classify did not write, is none)
    return (z < 0.0f && b >= MAX_BODIES && b < 2u * MAX_BODIES) ? b - MAX_BODIES : NONE;
}
// exactParts, exactValue (common.wgsl:1378-1412)
__device__ __forceinline__ void exactParts(float x, float scale, uint32_t* lo, uint32_t* hi) {
    const float s = rnd_even(clampf(x * scale, -9.2e18f, 9.2e18f));
    if (fabsf(s) < 2147483648.0f) {
        const int32_t v = f2i(s);
        *lo = (uint32_t)v;
        *hi = v < 0 ? 0xffffffffu : 0u;
        return;
    }
    const float h = floorf(s / 4294967296.0f);
    *lo = f2u(s - h * 4294967296.0f);
    *hi = (uint32_t)f2i(h);
}
__device__ __forceinline__ float exactValue(uint32_t lo, uint32_t hi, float scale) {
    const int32_t l = (int32_t)lo, h = (int32_t)hi;
    if ((h == 0 && l >= 0) || (h == -1 && l < 0)) return __int2float_rn(l) / scale;
    return (__int2float_rn(h) * 4294967296.0f + __uint2float_rn(lo)) / scale;
}
// pushSlot, addPush, pushOf (fluid.wgsl:1318-1338)
__device__ __forceinline__ uint32_t pushSlot(uint32_t b, uint32_t which, uint32_t k) {
    return b * WIG_BODY_PUSH_WORDS + 6u * which + 2u * k;
}
__device__ inline void addPush(const W& w, uint32_t b, uint32_t which, V3 v) {
    const float c[3] = {v.x, v.y, v.z};
    for (uint32_t k = 0; k < 3; k++) {
        uint32_t lo, hi;
        exactParts(c[k], EXACT_COARSE, &lo, &hi);
        uint32_t* at = w.D.pushes + pushSlot(b, which, k);
        const uint32_t old = atomicAdd(at, lo);
        atomicAdd(at + 1, hi + (old + lo < old ? 1u : 0u));
    }
}
__device__ inline V3 pushOf(const W& w, uint32_t b, uint32_t which) {
    const uint32_t* at = w.D.pushes + pushSlot(b, which, 0u);
    return V3{exactValue(at[0], at[1], EXACT_COARSE), exactValue(at[2], at[3], EXACT_COARSE),
              exactValue(at[4], at[5], EXACT_COARSE)};
}
// giveWay, pushChange, pushChangeFree (fluid.wgsl:1348-1372)
__device__ inline V3 giveWay(const W& w, uint32_t b, V3 g) {
    if (bodyWord(w, b, WIG_BW_MOBILITY_AT) != w.D.st->P.frame - 1u)
        return V3{g.x / rigidMass(w, b), g.y / rigidMass(w, b), g.z / rigidInertia(w, b)};
    float m[6];
    for (uint32_t k = 0; k < 6; k++) m[k] = bodyF(w, b, WIG_BW_MOBILITY + k);
    return V3{m[0] * g.x + m[1] * g.y + m[2] * g.z, m[1] * g.x + m[3] * g.y + m[4] * g.z,
              m[2] * g.x + m[4] * g.y + m[5] * g.z};
}
__device__ __forceinline__ V3 pushChange(const W& w, uint32_t b, uint32_t which) { return giveWay(w, b, pushOf(w, b, which)); }
__device__ inline V3 pushChangeFree(const W& w, uint32_t b, uint32_t which) {
    const V3 g = pushOf(w, b, which);
    return V3{g.x / rigidMass(w, b), g.y / rigidMass(w, b), g.z / rigidInertia(w, b)};
}
// bodyFaceJ (fluid.wgsl:1374-1379): the face from cell c to body b's cell q
__device__ inline V3 bodyFaceJ(const W& w, I2 c, I2 q, uint32_t b) {
    const V2 n{(float)(q.x - c.x), (float)(q.y - c.y)};
    const V2 pos = bodyV(w, b, WIG_BW_POS);
    const V2 r{(((float)c.x + 0.5f) + 0.5f * n.x) - pos.x, (((float)c.y + 0.5f) + 0.5f * n.y) - pos.y};
    return V3{n.x, n.y, r.x * n.y - r.y * n.x};
}
__device__ __forceinline__ V3 scale3(V3 v, float s) { return V3{v.x * s, v.y * s, v.z * s}; }
__device__ __forceinline__ V3 add3(V3 a, V3 b) { return V3{a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ float dot3(V3 a, V3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
// addPressurePush, couplingAt (fluid.wgsl:1381-1403)
__device__ inline void addPressurePush(const W& w, I2 c, float p, uint32_t which) {
    for (int d = 0; d < 4; d++) {
        const I2 q = beside(c, d);
        const uint32_t b = rigidAt(w, q);
        if (b != NONE) addPush(w, b, which, scale3(bodyFaceJ(w, c, q, b), p));
    }
}
__device__ inline float couplingAt(const W& w, I2 c, uint32_t which) {
    float sum = 0.0f;
    if (!w.D.motion) return sum;
    for (int d = 0; d < 4; d++) {
        const I2 q = beside(c, d);
        const uint32_t b = rigidAt(w, q);
        if (b != NONE) sum = sum + dot3(bodyFaceJ(w, c, q, b), pushChange(w, b, which));
    }
    return sum;
}
}  // namespace wig
