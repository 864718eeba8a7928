// direct.cu -- all-pairs Coulomb sum on GB300.
//
// Restates DirectForceFunction::direct (direct_force_method.cpp:153-190) and
// its rotational (direct_force_method_rotational.cpp:48-94) and translational
// (direct_force_method_translational.cpp:320-367) variants:
//     a_i = K q_i / m_i * sum_j q_j (r_i - r_j) / (|r_i - r_j|^2 + eps^2)^{3/2}
// for inbound targets i and sources j with status 1 or 2 (j != i for the plain
// sum; the symmetric variants keep the self image, which contributes 0).
//
// Targets and sources are the Morton-sorted copy (sort.cu), or for few pairs
// the copy with the sources first.
//
// MIXED: every unordered pair once.  The particles form blocks of 32 R; a warp
// holds a block's coordinates and sums in registers (R particles per lane) and
// takes tiles of 32 particles of another block, one per lane, which travel
// around the lanes together with their own sums: after 32 steps every pair of
// the block and the tile has been met once and has added to both sides
// (F_ji = -F_ij up to the charges).  A pair of interactions then costs 16
// FP32-pipe operations and one reciprocal square root instead of 24 and two.
// Coordinates are FP32 offsets from the block's middle particle, formed from the
// FP32 hi + lo parts that the sort wrote by an exact subtraction and one
// rounding; where a tile comes within the block's extent, the parts that rounding
// left out are kept too and added to each difference (six operations more, in a
// few tiles per block), so that every pair's offset is rounded relative to its own
// length and not to the block's; a wide plume (kWide) keeps all bits of the FP64 positions in
// a third part.  The force error against FP64 is 1.2e-7 to 3e-7
// (relative L2 over plumes of 256 to 30,011 ions); coordinates rounded relative to
// a CTA's first target gave 3e-7 to 5.6e-6, set by each plume's closest pairs.
// The loop has no FP64 instruction (GB300 issues one FP64 warp instruction in 64
// clocks: conversions and FP64 sums per 256-source tile took 12 to 18 % of the
// one-sided kernel).  At most 128 sources' (or 256 targets') FP32 sums go to the
// FP64 accumulators in memory at once.
//
// FP64: the same pairing with every operation in FP64, or (symmetry images)
// one-sided tiles in shared memory; r^-3 is a FP32 rsqrt seed and a third-order
// correction in FP64.
//
// Measured per launch (serialised), against the one-sided kernels they
// replaced: mixed, 30,011 particles of two charges 381 -> 289 us, 16,384 of one
// charge 123 -> 99 us, 3,001 with 81 images 652 -> 232 us (144 CTAs before: the
// images were not split); FP64, 4,096 particles 773 -> 285 us.
#include <algorithm>

#include "pairs.cuh"

namespace sv {
namespace {

// one-sided FP64 kernel (symmetry images)
constexpr int kTPB = 128;   // threads per CTA
constexpr int kTPT = 2;     // targets per thread
constexpr int kTile = 256;  // sources per shared-memory tile

struct Images {
    int kind;          // 0 none, 1 rotational (4 quadrants), 2 offsets
    int count;         // images per source
    const double *off; // device, 3*count metres (kind 2)
};

__device__ __forceinline__ void image_of(const Images &im, int g, double &x, double &y, double &z) {
    if (im.kind == 1) {
        // source rotated by g*pi/2 about z (quadrantRotationFunction, auxiliary_functions.h:55-57)
        const double x0 = x, y0 = y;
        if (g == 1) { x = -y0; y = x0; }
        else if (g == 2) { x = -x0; y = -y0; }
        else if (g == 3) { x = y0; y = -x0; }
    } else if (im.kind == 2) {
        // target shifted by -offset == source shifted by +offset
        x += im.off[3 * g];
        y += im.off[3 * g + 1];
        z += im.off[3 * g + 2];
    }
}

// true when any of the CTA's kTPB*kTPT targets has a nonzero K q/m (a target)
__device__ __forceinline__ bool block_has_target(const double *__restrict__ qm, int t0, int n) {
    int any = 0;
#pragma unroll
    for (int k = 0; k < kTPT; k++) {
        const int i = t0 + threadIdx.x + k * kTPB;
        any |= (i < n && qm[i] != 0.0);
    }
    return __syncthreads_or(any) != 0;
}

// ------------------------------------------------------------------ mixed --
struct PairArgs {
    const float4 *ph, *pl;   // sorted positions hi (w: charge) and lo (w: 1 = target)
    const float4 *pr;        // what hi and lo leave out (wide plumes)
    int n, nb;               // particles, blocks of 32 R of them
    int ct, nch;             // tiles per unit (of the R x images of a block pair), units per block pair
    float eps2;
    int kind, images;        // symmetry images, as Images
    const float4 *off;       // translational offsets: hi, lo and what they leave out (xyz) per image
    double *ax, *ay, *az;    // sums, added into
    const int *marks;        // nonzero: [0] source charges differ, [1] the plume is wide (kWide)
};

// A block's particles in registers (two per packed value) and the travelling
// particle; the parts of the block's coordinates below FP32 in shared memory (wide
// plumes: two of them).
template <int R>
struct PairBlock {
    float2 X[R / 2], Y[R / 2], Z[R / 2], Q[R / 2];   // coordinates, charges
    float2 gx[R / 2], gy[R / 2], gz[R / 2];          // sums
};
template <int R>
struct PairLow {
    float2 x[R / 2][32], y[R / 2][32], z[R / 2][32];
    float2 rx[R / 2][32], ry[R / 2][32], rz[R / 2][32];
};

// 32 steps of a travelling tile: negated coordinates (nx, ny, nz; what they leave out: m, k)
// and charge q; (sx, sy, sz) return the sums on the travelling particle (SYM).  (As three
// Parts the loop takes a move more per step: 2,000 particles with 81 images 185 -> 191 us.)
template <int R, bool UQ, bool CLAMP, bool SYM, int MODE>
__device__ __forceinline__ void pair_tile(PairBlock<R> &b, const PairLow<R> &low, float2 E2, float nx, float ny, float nz, float q,
                                          float mx, float my, float mz, float kx, float ky, float kz, float &sx, float &sy, float &sz) {
    auto dup = [](float v) { return make_float2(v, v); };
    constexpr int H = R / 2;
    const int lane = threadIdx.x & 31, from = (lane + 1) & 31;
#pragma unroll 1
    for (int step = 0; step < 32; step++) {
        const float2 NX = dup(nx), NY = dup(ny), NZ = dup(nz), QJ = dup(q);
        float2 jx, jy, jz;
#pragma unroll
        for (int p = 0; p < H; p++) {
            float2 dx = __fadd2_rn(b.X[p], NX), dy = __fadd2_rn(b.Y[p], NY), dz = __fadd2_rn(b.Z[p], NZ);
            if (MODE != kTileFar) {
                float2 ex = __fadd2_rn(low.x[p][lane], dup(mx)), ey = __fadd2_rn(low.y[p][lane], dup(my)),
                       ez = __fadd2_rn(low.z[p][lane], dup(mz));
                if (MODE == kTileWide) {
                    ex = __fadd2_rn(ex, __fadd2_rn(low.rx[p][lane], dup(kx)));
                    ey = __fadd2_rn(ey, __fadd2_rn(low.ry[p][lane], dup(ky)));
                    ez = __fadd2_rn(ez, __fadd2_rn(low.rz[p][lane], dup(kz)));
                }
                dx = __fadd2_rn(dx, ex);
                dy = __fadd2_rn(dy, ey);
                dz = __fadd2_rn(dz, ez);
            }
            float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, E2)));
            if (CLAMP) r2 = make_float2(fmaxf(r2.x, kMinR2), fmaxf(r2.y, kMinR2));
            const float2 inv = make_float2(rsqrt_ftz(r2.x), rsqrt_ftz(r2.y));
            const float2 w = __fmul2_rn(__fmul2_rn(inv, inv), inv);
            const float2 wi = UQ ? w : __fmul2_rn(QJ, w);
            b.gx[p] = __ffma2_rn(dx, wi, b.gx[p]);
            b.gy[p] = __ffma2_rn(dy, wi, b.gy[p]);
            b.gz[p] = __ffma2_rn(dz, wi, b.gz[p]);
            if (SYM) {
                const float2 wj = UQ ? w : __fmul2_rn(b.Q[p], w);
                jx = p == 0 ? __fmul2_rn(dx, wj) : __ffma2_rn(dx, wj, jx);
                jy = p == 0 ? __fmul2_rn(dy, wj) : __ffma2_rn(dy, wj, jy);
                jz = p == 0 ? __fmul2_rn(dz, wj) : __ffma2_rn(dz, wj, jz);
            }
        }
        nx = __shfl_sync(0xffffffffu, nx, from);
        ny = __shfl_sync(0xffffffffu, ny, from);
        nz = __shfl_sync(0xffffffffu, nz, from);
        if (MODE != kTileFar) {
            mx = __shfl_sync(0xffffffffu, mx, from);
            my = __shfl_sync(0xffffffffu, my, from);
            mz = __shfl_sync(0xffffffffu, mz, from);
        }
        if (MODE == kTileWide) {
            kx = __shfl_sync(0xffffffffu, kx, from);
            ky = __shfl_sync(0xffffffffu, ky, from);
            kz = __shfl_sync(0xffffffffu, kz, from);
        }
        if (!UQ) q = __shfl_sync(0xffffffffu, q, from);
        if (SYM) {
            sx = __shfl_sync(0xffffffffu, sx - (jx.x + jx.y), from);
            sy = __shfl_sync(0xffffffffu, sy - (jy.x + jy.y), from);
            sz = __shfl_sync(0xffffffffu, sz - (jz.x + jz.y), from);
        }
    }
}

// One unit: block A (registers) against tiles [k0, k1) of block B.  SYM: both
// sides' sums (A != B); otherwise the sums of A only (A == B, every ordered
// pair).  UQ: all charges equal, applied once at the end.
template <int R, bool UQ, bool CLAMP, bool SYM, bool WIDE>
__device__ __forceinline__ void pair_unit(const PairArgs &a, PairLow<R> &low, int A, int B, int k0, int k1) {
    const int lane = threadIdx.x & 31;
    const int i0 = A * 32 * R;
    const int io = min(i0 + 16 * R, a.n - 1);  // the block's middle particle: offsets half as long as from its first
    const float4 oh = a.ph[io], ol = a.pl[io];
    Parts ox{oh.x, ol.x}, oy{oh.y, ol.y}, oz{oh.z, ol.z};
    PairBlock<R> b;
    int tgt = 0;     // bit r: this lane's particle r of the block is a target
    float ext = 0.f;  // the block's largest offset on any axis
    __syncwarp();    // the previous unit's reads of `low`
    if (WIDE) {
        const float4 r = a.pr[io];
        ox.rest = r.x;
        oy.rest = r.y;
        oz.rest = r.z;
    }
#pragma unroll
    for (int p = 0; p < R / 2; p++) {
        Parts x[2], y[2], z[2];
        float c[2] = {0.f, 0.f};
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int i = i0 + 32 * (2 * p + u) + lane;
            if (i < a.n) {
                const float4 h = a.ph[i], l = a.pl[i], r = WIDE ? a.pr[i] : make_float4(0.f, 0.f, 0.f, 0.f);
                x[u] = parts_diff<WIDE>(Parts{h.x, l.x, r.x}, ox);
                y[u] = parts_diff<WIDE>(Parts{h.y, l.y, r.y}, oy);
                z[u] = parts_diff<WIDE>(Parts{h.z, l.z, r.z}, oz);
                c[u] = h.w;
                tgt |= l.w != 0.f ? 1 << (2 * p + u) : 0;
                ext = fmaxf(ext, fmaxf(fabsf(x[u].v), fmaxf(fabsf(y[u].v), fabsf(z[u].v))));
            } else {
                x[u].v = -kFar;
            }
        }
        b.X[p] = make_float2(x[0].v, x[1].v);
        b.Y[p] = make_float2(y[0].v, y[1].v);
        b.Z[p] = make_float2(z[0].v, z[1].v);
        b.Q[p] = make_float2(c[0], c[1]);
        low.x[p][lane] = make_float2(x[0].low, x[1].low);
        low.y[p][lane] = make_float2(y[0].low, y[1].low);
        low.z[p][lane] = make_float2(z[0].low, z[1].low);
        if (WIDE) {
            low.rx[p][lane] = make_float2(x[0].rest, x[1].rest);
            low.ry[p][lane] = make_float2(y[0].rest, y[1].rest);
            low.rz[p][lane] = make_float2(z[0].rest, z[1].rest);
        }
        b.gx[p] = b.gy[p] = b.gz[p] = make_float2(0.f, 0.f);
    }
    __syncwarp();
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ext = fmaxf(ext, __shfl_xor_sync(0xffffffffu, ext, o));
    const bool anyA = __any_sync(0xffffffffu, tgt);
    const float q0 = UQ ? oh.w : 1.f;
    const float2 E2 = make_float2(a.eps2, a.eps2);
    for (int k = k0; k < k1; k++) {
        const int g = k / R, j = B * 32 * R + 32 * (k - g * R) + lane;
        Parts x{kFar}, y, z;
        float q = 0.f;
        bool jt = false;
        if (j < a.n) {
            const float4 h = a.ph[j], l = a.pl[j], r = WIDE ? a.pr[j] : make_float4(0.f, 0.f, 0.f, 0.f);
            jt = l.w != 0.f;
            q = h.w;
            Parts px{h.x, l.x, r.x}, py{h.y, l.y, r.y}, pz{h.z, l.z, r.z}, cx = ox, cy = oy, cz = oz;
            if (a.kind == 1 && g) {
                // source rotated by g*pi/2 about z (quadrantRotationFunction, auxiliary_functions.h:55-57)
                const Parts x0 = px, y0 = py;
                px = g == 1 ? negated(y0) : g == 2 ? negated(x0) : y0;
                py = g == 1 ? x0 : g == 2 ? negated(y0) : negated(x0);
            } else if (a.kind == 2) {
                // source shifted by the image offset: the origin shifted back
                const float4 fh = a.off[3 * g], fl = a.off[3 * g + 1],
                             fr = WIDE ? a.off[3 * g + 2] : make_float4(0.f, 0.f, 0.f, 0.f);
                auto back = [](const Parts &o, const Parts &f) {
                    if (WIDE) return parts_diff<WIDE>(o, f);
                    const float s = o.v - f.v, bb = s - o.v;
                    const float e = ((o.v - (s - bb)) - (f.v + bb)) + (o.low - f.low), r = s + e;
                    return Parts{r, e - (r - s)};
                };
                cx = back(cx, Parts{fh.x, fl.x, fr.x});
                cy = back(cy, Parts{fh.y, fl.y, fr.y});
                cz = back(cz, Parts{fh.z, fl.z, fr.z});
            }
            x = parts_diff<WIDE>(px, cx);
            y = parts_diff<WIDE>(py, cy);
            z = parts_diff<WIDE>(pz, cz);
        }
        // within twice the block's extent of its origin (a pair may be closer than
        // the coordinates' rounding allows for)
        const bool near = j < a.n && fmaxf(fabsf(x.v), fmaxf(fabsf(y.v), fabsf(z.v))) <= 2.f * ext;
        const bool anyB = SYM && __any_sync(0xffffffffu, jt);
        if (!anyA && !anyB) continue;
        float sx = 0.f, sy = 0.f, sz = 0.f;  // the travelling particle's sums
        if (!SYM || __any_sync(0xffffffffu, near)) {
            pair_tile<R, UQ, CLAMP, SYM, WIDE ? kTileWide : kTileNear>(b, low, E2, -x.v, -y.v, -z.v, q, -x.low, -y.low, -z.low, -x.rest, -y.rest, -z.rest, sx, sy, sz);
        } else pair_tile<R, UQ, CLAMP, SYM, kTileFar>(b, low, E2, -x.v, -y.v, -z.v, q, -x.low, -y.low, -z.low, -x.rest, -y.rest, -z.rest, sx, sy, sz);
        if (SYM && jt) {
            if (a.kind == 1 && g) {  // the sum on the unrotated particle: turned back by -g*pi/2
                const float tx = sx, ty = sy;
                if (g == 2) {
                    sx = -tx;
                    sy = -ty;
                } else {
                    sx = g == 1 ? ty : -ty;
                    sy = g == 1 ? -tx : tx;
                }
            }
            atomicAdd(&a.ax[j], widen(sx * q0));
            atomicAdd(&a.ay[j], widen(sy * q0));
            atomicAdd(&a.az[j], widen(sz * q0));
        }
    }
    if (!anyA) return;
#pragma unroll
    for (int r = 0; r < R; r++) {
        if (!(tgt >> r & 1)) continue;
        const int i = i0 + 32 * r + lane;
        atomicAdd(&a.ax[i], widen((r & 1 ? b.gx[r / 2].y : b.gx[r / 2].x) * q0));
        atomicAdd(&a.ay[i], widen((r & 1 ? b.gy[r / 2].y : b.gy[r / 2].x) * q0));
        atomicAdd(&a.az[i], widen((r & 1 ? b.gz[r / 2].y : b.gz[r / 2].x) * q0));
    }
}

// All units of a warp of a wide plume, with any charges: out of line and called once, for
// its code beside the other's costs the other plumes (per launch, without it / so / in
// line: 4,096 particles 15.5 / 15.8 / 18.2 us, 16,384 97 / 99 / 102).
template <int R, bool CLAMP>
__device__ __noinline__ void pairs_wide(PairArgs a, PairLow<R> &low, int64_t v) {
    for (int d = blockIdx.y; d <= a.nb / 2; d += gridDim.y) {
        int A, B, ch;
        if (!unit_blocks(v, d, a.nb, a.nch, A, B, ch)) return;
        const int k0 = ch * a.ct, k1 = min(k0 + a.ct, R * a.images);
        if (A != B) pair_unit<R, false, CLAMP, true, true>(a, low, A, B, k0, k1);
        else pair_unit<R, false, CLAMP, false, true>(a, low, A, B, k0, k1);
    }
}

template <int R, bool CLAMP>
__global__ void __launch_bounds__(32 * kPairWarps, 3) direct_pairs_kernel(PairArgs a) {
    __shared__ PairLow<R> lows[kPairWarps];
    PairLow<R> &low = lows[threadIdx.x >> 5];
    const int64_t v = (int64_t)blockIdx.x * kPairWarps + (threadIdx.x >> 5);
    if (a.marks[1] != 0) {
        pairs_wide<R, CLAMP>(a, low, v);
        return;
    }
    const bool differ = a.marks[0] != 0;
    for (int d = blockIdx.y; d <= a.nb / 2; d += gridDim.y) {
        int A, B, ch;
        if (!unit_blocks(v, d, a.nb, a.nch, A, B, ch)) return;  // also for every larger distance
        const int k0 = ch * a.ct, k1 = min(k0 + a.ct, R * a.images);
        if (differ) {
            if (A != B) pair_unit<R, false, CLAMP, true, false>(a, low, A, B, k0, k1);
            else pair_unit<R, false, CLAMP, false, false>(a, low, A, B, k0, k1);
        } else {
            if (A != B) pair_unit<R, true, CLAMP, true, false>(a, low, A, B, k0, k1);
            else pair_unit<R, true, CLAMP, false, false>(a, low, A, B, k0, k1);
        }
    }
}

template <int R>
cudaError_t launch_pairs(PairArgs a, cudaStream_t st) {
    a.nb = div_up(a.n, 32 * R);
    // about 16 units per SM sub-partition, of at most kMaxTiles tiles
    const int64_t per = (int64_t)R * a.images, tiles = ((int64_t)a.nb * (a.nb + 1) / 2) * per;
    a.ct = (int)std::max<int64_t>(1, std::min<int64_t>(kMaxTiles, tiles / (64 * (int64_t)device_sms())));
    a.nch = div_up(per, a.ct);
    const dim3 grid = pair_grid(a.nb, a.nch);
    if (a.eps2 >= kMinR2) direct_pairs_kernel<R, false><<<grid, 32 * kPairWarps, 0, st>>>(a);
    else direct_pairs_kernel<R, true><<<grid, 32 * kPairWarps, 0, st>>>(a);
    return cudaGetLastError();
}

// R = 8 amortises the travelling particle's shuffles over eight pairs; below
// 2,048 particles its few units would leave most of the GPU idle
cudaError_t launch_pairs(const PairArgs &a, cudaStream_t st) {
    if (a.n <= 0) return cudaSuccess;
    return a.n < 2048 ? launch_pairs<2>(a, st) : launch_pairs<8>(a, st);
}

// ------------------------------------------------------------------- FP64 --
// r2^(-3/2) in FP64: y^3 (1 - e)^(-3/2) from rsqrt_seed_f64's y with e = 1 - r2 y^2,
// to second order in e (the next term is below 2e-19): six FP64 operations, where
// two Newton steps on 1/r and its cube took nine and two conversions at the FP64
// rate.
__device__ __forceinline__ double inv_cube_f64(double r2) {
    const double y = rsqrt_seed_f64(r2);
    const double y2 = y * y, e = fma(-r2, y2, 1.0), y3 = y2 * y;
    return fma(y3 * e, fma(1.875, e, 1.5), y3);
}

struct Pair64Args {
    const double *x, *y, *z, *qm;
    const float *q;
    int n, nb;
    double eps2;
    double *ax, *ay, *az;
};

// Every unordered pair once, as the mixed kernel: one particle per lane against
// a tile of 32 that travels around the lanes with its sums.  FP64-pipe bound: 20
// operations per pair of interactions, 18 where the charges of both tiles are equal
// (UQ) and are applied once after the tile; shuffles, loads and atomics are free
// beside them.
template <bool UQ, bool SYM>
__device__ __forceinline__ void pair64_tile(double xi, double yi, double zi, double qi, double xj, double yj,
                                            double zj, double qj, double eps2, double (&f)[3], double (&g)[3]) {
    const int from = ((threadIdx.x & 31) + 1) & 31;
#pragma unroll 2
    for (int step = 0; step < 32; step++) {
        const double dx = xi - xj, dy = yi - yj, dz = zi - zj;
        const double w = inv_cube_f64(fma(dx, dx, fma(dy, dy, fma(dz, dz, eps2))));
        const double wi = UQ ? w : qj * w;
        f[0] = fma(dx, wi, f[0]);
        f[1] = fma(dy, wi, f[1]);
        f[2] = fma(dz, wi, f[2]);
        if (SYM) {
            const double wj = UQ ? -w : -(qi * w);
            g[0] = __shfl_sync(0xffffffffu, fma(dx, wj, g[0]), from);
            g[1] = __shfl_sync(0xffffffffu, fma(dy, wj, g[1]), from);
            g[2] = __shfl_sync(0xffffffffu, fma(dz, wj, g[2]), from);
        }
        xj = __shfl_sync(0xffffffffu, xj, from);
        yj = __shfl_sync(0xffffffffu, yj, from);
        zj = __shfl_sync(0xffffffffu, zj, from);
        if (!UQ) qj = __shfl_sync(0xffffffffu, qj, from);
    }
}

template <bool SYM>
__device__ __forceinline__ void pair64_unit(const Pair64Args &a, int A, int B) {
    const int lane = threadIdx.x & 31, i = 32 * A + lane, j = 32 * B + lane;
    const int ii = min(i, a.n - 1), jj = min(j, a.n - 1);
    const bool it = i < a.n && a.qm[ii] != 0.0, jt = SYM && j < a.n && a.qm[jj] != 0.0;
    if (!__any_sync(0xffffffffu, it || jt)) return;
    // absent particles carry no charge
    const double qi = i < a.n ? (double)a.q[ii] : 0.0, qj = j < a.n ? (double)a.q[jj] : 0.0;
    const double q0 = __shfl_sync(0xffffffffu, qi, 0);
    const bool equal = __all_sync(0xffffffffu, qi == q0 && qj == q0);
    double f[3] = {0.0, 0.0, 0.0}, g[3] = {0.0, 0.0, 0.0};
    if (equal) pair64_tile<true, SYM>(a.x[ii], a.y[ii], a.z[ii], qi, a.x[jj], a.y[jj], a.z[jj], qj, a.eps2, f, g);
    else pair64_tile<false, SYM>(a.x[ii], a.y[ii], a.z[ii], qi, a.x[jj], a.y[jj], a.z[jj], qj, a.eps2, f, g);
    const double k = equal ? q0 : 1.0;
    if (it) {
        atomicAdd(&a.ax[i], f[0] * k);
        atomicAdd(&a.ay[i], f[1] * k);
        atomicAdd(&a.az[i], f[2] * k);
    }
    if (jt) {
        atomicAdd(&a.ax[j], g[0] * k);
        atomicAdd(&a.ay[j], g[1] * k);
        atomicAdd(&a.az[j], g[2] * k);
    }
}

__global__ void __launch_bounds__(32 * kPairWarps) direct_pairs64_kernel(Pair64Args a) {
    const int64_t v = (int64_t)blockIdx.x * kPairWarps + (threadIdx.x >> 5);
    for (int d = blockIdx.y; d <= a.nb / 2; d += gridDim.y) {
        int A, B, ch;
        if (!unit_blocks(v, d, a.nb, 1, A, B, ch)) return;
        if (A != B) pair64_unit<true>(a, A, B);
        else pair64_unit<false>(a, A, B);
    }
}

// One-sided FP64 sum with symmetry images: kTPB * kTPT targets per CTA against
// (image, source tile) units [blockIdx.y * per, + per).
__global__ void __launch_bounds__(kTPB)
direct_fp64_kernel(const double *__restrict__ xs, const double *__restrict__ ys,
                   const double *__restrict__ zs, const float *__restrict__ qs,
                   const double *__restrict__ qm, int n, int64_t per, double eps2, Images im,
                   double *__restrict__ ax, double *__restrict__ ay, double *__restrict__ az) {
    __shared__ dbl4_t tile[kTile];
    const int t0 = blockIdx.x * (kTPB * kTPT);
    const int ntile = (n + kTile - 1) / kTile;
    const int64_t u0 = blockIdx.y * per, u1 = min(u0 + per, (int64_t)ntile * im.count);
    double tx[kTPT], ty[kTPT], tz[kTPT], sx[kTPT], sy[kTPT], sz[kTPT];
    if (!block_has_target(qm, t0, n)) return;
#pragma unroll
    for (int k = 0; k < kTPT; k++) {
        const int ii = min(t0 + (int)threadIdx.x + k * kTPB, n - 1);
        tx[k] = xs[ii];
        ty[k] = ys[ii];
        tz[k] = zs[ii];
        sx[k] = sy[k] = sz[k] = 0.0;
    }
    for (int64_t u = u0; u < u1; u++) {
        const int g = (int)(u / ntile), jt = (int)(u - (int64_t)g * ntile) * kTile;
        __syncthreads();
        for (int s = threadIdx.x; s < kTile; s += kTPB) {
            const int j = min(jt + s, n - 1);
            double px = xs[j], py = ys[j], pz = zs[j];
            image_of(im, g, px, py, pz);
            tile[s] = dbl4(px, py, pz, jt + s < n ? (double)qs[j] : 0.0);
        }
        __syncthreads();
#pragma unroll 2
        for (int s = 0; s < kTile; s++) {
            const dbl4_t v = tile[s];
#pragma unroll
            for (int k = 0; k < kTPT; k++) {
                const double dx = tx[k] - v.x, dy = ty[k] - v.y, dz = tz[k] - v.z;
                const double w = v.w * inv_cube_f64(fma(dx, dx, fma(dy, dy, fma(dz, dz, eps2))));
                sx[k] = fma(dx, w, sx[k]);
                sy[k] = fma(dy, w, sy[k]);
                sz[k] = fma(dz, w, sz[k]);
            }
        }
    }
#pragma unroll
    for (int k = 0; k < kTPT; k++) {
        const int i = t0 + threadIdx.x + k * kTPB;
        if (i >= n || qm[i] == 0.0) continue;
        atomicAdd(&ax[i], sx[k]);
        atomicAdd(&ay[i], sy[k]);
        atomicAdd(&az[i], sz[k]);
    }
}

}  // namespace

void direct_sort_wants(sv_ctx *c) {
    c->S.want.zero = true;
    c->S.want.hilo = c->P.precision == SV_PREC_MIXED;
    c->S.want.rest = c->S.want.hilo;
    c->S.want.hl_abs = c->P.symmetry == SV_SYM_ROTATIONAL;
    const ImageSet *I = nullptr;
    int64_t images = c->P.symmetry == SV_SYM_ROTATIONAL ? 4 : 1;
    if (c->P.symmetry == SV_SYM_TRANSLATIONAL) images = image_set(c, &I) == SV_OK ? I->count : INT32_MAX;
    c->S.want.any_order = c->n * c->n <= kAnyOrderMax * kAnyOrderMax / images;
}

sv_status direct_accel(sv_ctx *c) {
    const int n = (int)c->S.n;
    Sorted &S = c->S;
    Images im{0, 1, nullptr};
    const float4 *off_hl = nullptr;
    if (c->P.symmetry == SV_SYM_ROTATIONAL) {
        im.kind = 1;
        im.count = 4;
    } else if (c->P.symmetry == SV_SYM_TRANSLATIONAL) {
        const ImageSet *I = nullptr;
        SV_TRY(image_set(c, &I));
        im.kind = 2;
        im.count = I->count;
        im.off = I->m;
        off_hl = I->hl;
    }
    for (int k = 2; k <= 6; k++) phase_mark(c, k);
    S.raw = true;
    if (c->P.precision == SV_PREC_FP64 && im.kind == 0) {
        const Pair64Args a{S.x, S.y, S.z, S.qm, S.q, n, div_up(n, 32), c->P.softening2, S.ax, S.ay, S.az};
        direct_pairs64_kernel<<<pair_grid(a.nb, 1), 32 * kPairWarps, 0, c->stream>>>(a);
    } else if (c->P.precision == SV_PREC_FP64) {
        // the (image, tile) units split so that the grid fills the GPU ~8 CTAs per SM deep
        const int tblocks = div_up(n, kTPB * kTPT);
        const int64_t units = (int64_t)div_up(n, kTile) * im.count;
        const int64_t splits = std::max<int64_t>(1, std::min<int64_t>({div_up(8 * device_sms(), tblocks), units, 65535}));
        const int64_t per = (units + splits - 1) / splits;
        direct_fp64_kernel<<<dim3(tblocks, (unsigned)div_up(units, per)), kTPB, 0, c->stream>>>(
            S.x, S.y, S.z, S.q, S.qm, n, per, c->P.softening2, im, S.ax, S.ay, S.az);
    } else {
        PairArgs a{};
        a.ph = S.ph;
        a.pl = S.pl;
        a.n = n;
        a.eps2 = (float)c->P.softening2;
        a.kind = im.kind;
        a.images = im.count;
        a.off = off_hl;
        a.pr = S.pr;
        a.ax = S.ax;
        a.ay = S.ay;
        a.az = S.az;
        a.marks = reinterpret_cast<const int *>(S.root + 14);
        SV_CK(c, launch_pairs(a, c->stream));
    }
    SV_LAUNCHED(c);
    const double pairs = (double)n * (double)n * (double)im.count;
    c->stats.pair_interactions = pairs;
    c->stats.cell_interactions = 0;
    c->stats.flops_algorithmic = 20.0 * pairs;
    return SV_OK;
}

cudaError_t launch_direct_mixed_sorted(const float4 *ph, const float4 *pl, const float4 *pr, int n, float eps2,
                                       double *ax, double *ay, double *az, const int *marks, cudaStream_t stream) {
    PairArgs a{};
    a.ph = ph;
    a.pl = pl;
    a.pr = pr;
    a.n = n;
    a.eps2 = eps2;
    a.images = 1;
    a.ax = ax;
    a.ay = ay;
    a.az = az;
    a.marks = marks;
    return launch_pairs(a, stream);
}

}  // namespace sv
