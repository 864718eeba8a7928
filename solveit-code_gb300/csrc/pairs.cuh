// pairs.cuh -- pieces shared by the kernels that visit every unordered pair of
// particles once (direct.cu, adjoint.cu): the particles form blocks, a warp holds
// one block in registers and a tile of 32 particles of another block travels
// around its lanes with its own sums.
#pragma once

#include <algorithm>

#include "sv_internal.cuh"

namespace sv {

// (hi + lo) - (ohi + olo) as r + res: r the difference rounded once (of the hi
// parts with its exact rounding error, Knuth, then the small parts), res what
// that rounding left out
__device__ __forceinline__ float hilo_diff(float hi, float lo, float ohi, float olo, float &res) {
    const float s = hi - ohi, bb = s - hi;
    const float t = ((hi - (s - bb)) - (ohi + bb)) + (lo - olo);
    const float r = s + t, tt = r - s;
    res = (s - (r - tt)) + (t - tt);
    return r;
}

// a float's value as a double, by its bits (the conversion instruction runs at
// the FP64 rate); denormals become zero
__device__ __forceinline__ double widen(float f) {
    const uint32_t u = __float_as_uint(f), m = u & 0x7fffffffu;
    uint32_t hi = (m >> 3) + 0x38000000u, lo = u << 29;
    if (m >= 0x7f800000u) hi |= 0x7ff00000u;
    if (m < 0x00800000u) hi = lo = 0;
    return __hiloint2double((int)(hi | (u & 0x80000000u)), (int)lo);
}

// v as FP32 hi (truncated, by bits) + lo parts: one FP64 subtraction and one
// conversion instead of four operations at the FP64 rate
__device__ __forceinline__ void split_hilo_bits(double v, float &hi, float &lo) {
    const uint32_t vh = (uint32_t)__double2hiint(v), m = vh & 0x7fffffffu;
    if (m < 0x38100000u || m >= 0x47f00000u) {  // outside FP32's normal range
        split_hilo(v, hi, lo);
        return;
    }
    hi = __uint_as_float((vh & 0x80000000u) | ((m - 0x38000000u) << 3) | ((uint32_t)__double2loint(v) >> 29));
    lo = (float)(v - widen(hi));
}

// A coordinate as FP32 parts: the value rounded once, what that left out, and (wide
// plumes) what both left out.
struct Parts {
    float v = 0.f, low = 0.f, rest = 0.f;
};
__device__ __forceinline__ Parts negated(const Parts &p) { return Parts{-p.v, -p.low, -p.rest}; }

// a + b as its rounded value and the exact rest (Knuth)
__device__ __forceinline__ float two_sum(float a, float b, float &err) {
    const float s = a + b, bb = s - a;
    err = (a - (s - bb)) + (b - bb);
    return s;
}

// The difference a - o of two coordinates as parts that do not overlap: of the first
// two parts with hilo_diff, or (wide) of all three, exact to their last bits.
template <bool WIDE>
__device__ __forceinline__ Parts parts_diff(const Parts &a, const Parts &o) {
    Parts d;
    if (!WIDE) {
        d.v = hilo_diff(a.v, a.low, o.v, o.low, d.low);
        return d;
    }
    float e, f, g, h;
    const float s = two_sum(a.v, -o.v, e), t = two_sum(a.low, -o.low, f);
    const float u = two_sum(e, t, g);
    d.v = two_sum(s, u, h);
    const float r = g + (f + (a.rest - o.rest));
    d.low = h + r;
    d.rest = r - (d.low - h);
    return d;
}

// Tiles by distance: far from the block, near it (the second parts added to each
// difference), of a wide plume (all three: the FP64 difference, rounded to FP32)
enum { kTileFar, kTileNear, kTileWide };

constexpr int kPairWarps = 4;    // warps (units) per CTA
constexpr int kMaxTiles = 4;     // tiles per unit: 128 sources per FP32 sum of a target
constexpr float kFar = 1e18f;    // coordinate of absent particles: r^-3 underflows to zero

// 1/sqrt(r2) to FP32 precision as a double (relative error e/2 with |e| < 4e-7,
// e = 1 - r2 y^2): the FP32 reciprocal square root of the truncated r2, converted
// by bits on the integer pipe (the conversion instructions run at the FP64
// rate).  r2 past the FP32 range gives 0, below it the smallest normal seed (a
// zero distance stays finite).
__device__ __forceinline__ double rsqrt_seed_f64(double r2) {
    const int h = max(__double2hiint(r2), 0x38100000);
    const int f = h >= 0x47f00000 ? 0x7f800000 : (int)(((uint32_t)(h - 0x38000000) << 3) |
                                                       ((uint32_t)__double2loint(r2) >> 29));
    const uint32_t u = __float_as_uint(rsqrt_ftz(__int_as_float(f)));
    return u ? __hiloint2double((int)((u >> 3) + 0x38000000u), (int)(u << 29)) : 0.0;
}

// Unit (v, d) -> block pair (A, A + d mod nb), d = 0 .. nb / 2 (for even nb the
// last distance from the first half of the blocks only): every unordered block
// pair once.
__device__ __forceinline__ bool unit_blocks(int64_t v, int d, int nb, int nch, int &A, int &B, int &ch) {
    A = (int)(v / nch);
    ch = (int)(v - (int64_t)A * nch);
    if (A >= nb || (2 * (int64_t)d == nb && 2 * (int64_t)A >= nb)) return false;
    B = (int)(((int64_t)A + d) % nb);
    return true;
}
// grid of nb x nch units per distance, kPairWarps to a CTA; distances in y
inline dim3 pair_grid(int nb, int nch) {
    return dim3((unsigned)div_up((int64_t)nb * nch, kPairWarps), (unsigned)std::min(nb / 2 + 1, 65535));
}

}  // namespace sv
