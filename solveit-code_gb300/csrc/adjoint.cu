// adjoint.cu -- hand-written adjoint of the leapfrog DKD step and the direct sum.
//
// No counterpart in the reference (its integrator only runs forward,
// integration_schemes.cpp:856-891).  Forward step s (t_s = t0 + s dt),
// as sv_leapfrog runs it:
//     x_h     = x_s + h1 v_s                    h1 = clamp(t_s + dt/2 - t_inj, 0, dt/2)
//     a       = F(x_h) + c E                    c = (e/amu) q/m, F = direct sum
//     v_{s+1} = v_s + k a                       k  = clamp(t_s + dt - t_inj, 0, dt), status 1
//     x_{s+1} = x_h + h2 v_{s+1}                h2 = clamp(t_s + dt - t_inj, 0, dt/2)
// F and k act on the injection window t_inj <= t_s + dt/2 only (targets and
// sources); crash, boundary and folding steps are not differentiated (the
// adjoint refuses a context that has them on).
// Reverse step with adjoints (lx, lv) of (x_{s+1}, v_{s+1}):
//     lv += h2 lx;   lh = lx;   la = k lv;   lE += sum_i c_i la_i
//     lh += J(x_h)^T la;        lx = lh;     lv += h1 lh
// with the Jacobian-transpose product of the softened Coulomb sum
//     (J^T la)_k = sum_j G(x_k - x_j) (q_j u_k - q_k u_j),  u = K q/m la,
//     G(d) = I / s^3 - 3 d d^T / s^5,  s^2 = |d|^2 + eps^2,
// a pair kernel that visits every unordered pair once, as the direct sum's: the
// contribution to j is minus the contribution to k.
// The forward pass keeps the state every `checkpoint_every` steps and the x_h of
// its last segment; the backward pass re-runs each other segment from its
// checkpoint, keeping the segment's x_h, and walks it in reverse.
#include <cfloat>

#include "pairs.cuh"

namespace sv {

struct Adj {
    int nsteps = 0, every = 0, nck = 0;
    double dt = 0, t0 = 0;
    int64_t n = 0, cap = 0;
    int seg_cap = 0;
    int xh_seg = -1;          // segment whose x_h are in xh (-1: none that still holds)
    double *ck = nullptr;     // nck x 6 x n: x, y, z, vx, vy, vz
    double *xh = nullptr;     // every x 3 x n: x_h of a segment
    double *lam = nullptr;    // lx(3) lv(3) la(3) x n, then 4 n + 2: staging, or u as FP32 hi and lo float4s
    double *fin = nullptr;    // 6 x n: final state, restored after the backward pass
    double *lE = nullptr;     // 4: dL/dE, then max |u| scratch
    bool forward_done = false;
};

namespace {

__device__ __forceinline__ double clampd(double v, double hi) { return fmin(fmax(v, 0.0), hi); }

// Start of a reverse step at its mid positions xh (x, y, z of n each): the state's
// positions and the step's window; (1)-(4): lv += h2 lx; lh = lx (in place); la =
// k lv; lE += c la; and max |u| of u = K q/m la (non-negative doubles order like
// their bit patterns)
struct PrepArgs {
    const double *xh;
    double *x, *y, *z;
    int32_t *wst;
    const double *lx;       // lx, ly, lz of n each
    double *lv, *la;        // likewise
    const double *qom, *t_inj;
    const int32_t *st;
    int64_t n;
    double ts, dt, eoa, kconst;
    double *lE;
    unsigned long long *umax;
};

__global__ void adj_prep(PrepArgs a) {
    double e0 = 0, e1 = 0, e2 = 0, um = 0;
    const int64_t n = a.n;
    const double h = 0.5 * a.dt;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        a.x[i] = a.xh[i];
        a.y[i] = a.xh[n + i];
        a.z[i] = a.xh[2 * n + i];
        const int32_t w = a.st[i];
        const double ti = a.t_inj[i];
        const int32_t ws = ti <= a.ts + h ? w : 0;
        a.wst[i] = ws;
        const double h2 = (w == 1 || w == 2) ? clampd(a.ts + a.dt - ti, h) : 0.0;
        // kicked: inbound and injected by the step's mid time (the window of the force)
        const double k = ws == 1 ? clampd(a.ts + a.dt - ti, a.dt) : 0.0;
        const double vx = a.lv[i] + h2 * a.lx[i], vy = a.lv[n + i] + h2 * a.lx[n + i],
                     vz = a.lv[2 * n + i] + h2 * a.lx[2 * n + i];
        a.lv[i] = vx;
        a.lv[n + i] = vy;
        a.lv[2 * n + i] = vz;
        a.la[i] = k * vx;
        a.la[n + i] = k * vy;
        a.la[2 * n + i] = k * vz;
        const double c = w == 1 ? a.eoa * a.qom[i] : 0.0;
        e0 += c * k * vx;
        e1 += c * k * vy;
        e2 += c * k * vz;
        const double u = fabs(a.kconst * a.qom[i] * k) * fmax(fabs(vx), fmax(fabs(vy), fabs(vz)));
        if (u <= DBL_MAX) um = fmax(um, u);  // a non-finite adjoint propagates through the sum itself
    }
    for (int o = 16; o > 0; o >>= 1) {
        e0 += __shfl_xor_sync(0xffffffffu, e0, o);
        e1 += __shfl_xor_sync(0xffffffffu, e1, o);
        e2 += __shfl_xor_sync(0xffffffffu, e2, o);
        um = fmax(um, __shfl_xor_sync(0xffffffffu, um, o));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&a.lE[0], e0);
        atomicAdd(&a.lE[1], e1);
        atomicAdd(&a.lE[2], e2);
        if (um > 0.0) atomicMax(a.umax, (unsigned long long)__double_as_longlong(um));
    }
}

// the power of two that brings max |u| into [1/2, 1) (1 when it is zero), and
// the exponent it removes
__device__ __forceinline__ double u_scale(double um, int &ue) {
    ue = 0;
    if (um > 0.0) frexp(um, &ue);
    return ldexp(1.0, -ue);
}

constexpr double kLen = 1073741824.0;  // 2^30: mixed-precision coordinates are in 2^-30 m (1/s^5 in metres overflows FP32)

// u = K q/m la in sorted order (S.qm is K q/m for targets, 0 otherwise): FP64
// values, or scaled FP32 hi and lo parts
__global__ void adj_gather_u(const uint32_t *__restrict__ idx, int n, const double *__restrict__ qm,
                             const double *__restrict__ la, const double *__restrict__ umax,
                             double *__restrict__ u, float4 *__restrict__ uh, float4 *__restrict__ ul) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const uint32_t i = idx[s];
    const double k = qm[s];
    const double v[3] = {k * la[i], k * la[n + i], k * la[2 * (int64_t)n + i]};
    if (u) {
        for (int d = 0; d < 3; d++) u[d * (int64_t)n + s] = v[d];
        return;
    }
    int ue;
    const double su = u_scale(*umax, ue);
    float4 h = make_float4(0.f, 0.f, 0.f, 0.f), l = h;
    split_hilo(v[0] * su, h.x, l.x);
    split_hilo(v[1] * su, h.y, l.y);
    split_hilo(v[2] * su, h.z, l.z);
    uh[s] = h;
    ul[s] = l;
}

// End of a reverse step: lh += J^T la (the sorted sums, times their scale), then
// lx = lh, lv += h1 lh
__global__ void adj_post(const uint32_t *__restrict__ idx, int64_t n, const double *__restrict__ jx,
                         const double *__restrict__ jy, const double *__restrict__ jz, int mixed,
                         unsigned long long *__restrict__ umax, double *__restrict__ lx, double *__restrict__ lv,
                         const int32_t *__restrict__ st, const double *__restrict__ t_inj, double ts, double dt) {
    const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (s >= n) return;
    double back = 1.0;
    if (mixed) {
        int ue;
        (void)u_scale(__longlong_as_double((long long)*umax), ue);
        back = ldexp(1.0, 90 + ue);
    }
    const uint32_t i = idx[s];
    const double h = 0.5 * dt;
    const int32_t w = st[i];
    const double h1 = (w == 1 || w == 2) ? clampd(ts + h - t_inj[i], h) : 0.0;
    const double j[3] = {jx[s], jy[s], jz[s]};
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const double l = lx[d * n + i] + j[d] * back;
        lx[d * n + i] = l;
        lv[d * n + i] += h1 * l;
    }
}

// ------------------------------------------- Jacobian-transpose pair sums --
struct JPair64Args {
    const double *x, *y, *z, *u;  // u: x, y, z of n each
    const float *q;
    int n, nb;
    double eps2;
    double *ox, *oy, *oz;
};

// FP64: one particle per lane against a tile of 32 that travels around the lanes
// with its sums (SYM; otherwise every ordered pair of one block).
template <bool SYM>
__device__ __forceinline__ void jtv64_unit(const JPair64Args &a, int A, int B) {
    const int lane = threadIdx.x & 31, i = 32 * A + lane, j = 32 * B + lane;
    const int64_t n = a.n;
    const int ii = min(i, a.n - 1), jj = min(j, a.n - 1);
    const bool li = i < a.n, lj = j < a.n;  // absent particles carry neither charge nor adjoint
    const double xi = a.x[ii], yi = a.y[ii], zi = a.z[ii], qi = li ? (double)a.q[ii] : 0.0;
    const double uxi = li ? a.u[ii] : 0.0, uyi = li ? a.u[n + ii] : 0.0, uzi = li ? a.u[2 * n + ii] : 0.0;
    double xj = a.x[jj], yj = a.y[jj], zj = a.z[jj], qj = lj ? (double)a.q[jj] : 0.0;
    double uxj = lj ? a.u[jj] : 0.0, uyj = lj ? a.u[n + jj] : 0.0, uzj = lj ? a.u[2 * n + jj] : 0.0;
    double fx = 0.0, fy = 0.0, fz = 0.0, gx = 0.0, gy = 0.0, gz = 0.0;
    const int from = (lane + 1) & 31;
    for (int step = 0; step < 32; step++) {
        const double dx = xi - xj, dy = yi - yj, dz = zi - zj;
        const double r2 = fma(dx, dx, fma(dy, dy, fma(dz, dz, a.eps2)));
        // 1/s from the FP32 seed, to second order in e = 1 - r2 y^2
        const double y = rsqrt_seed_f64(r2), e = fma(-r2, y * y, 1.0);
        const double inv = fma(y * e, fma(0.375, e, 0.5), y);
        const double inv2 = inv * inv, inv3 = inv * inv2;
        const double wx = qj * uxi - qi * uxj, wy = qj * uyi - qi * uyj, wz = qj * uzi - qi * uzj;
        const double dw = -3.0 * (fma(dx, wx, fma(dy, wy, dz * wz)) * inv2) * inv3;
        const double vx = fma(dw, dx, wx * inv3), vy = fma(dw, dy, wy * inv3), vz = fma(dw, dz, wz * inv3);
        fx += vx;
        fy += vy;
        fz += vz;
        if (SYM) {
            gx = __shfl_sync(0xffffffffu, gx - vx, from);
            gy = __shfl_sync(0xffffffffu, gy - vy, from);
            gz = __shfl_sync(0xffffffffu, gz - vz, from);
        }
        xj = __shfl_sync(0xffffffffu, xj, from);
        yj = __shfl_sync(0xffffffffu, yj, from);
        zj = __shfl_sync(0xffffffffu, zj, from);
        qj = __shfl_sync(0xffffffffu, qj, from);
        uxj = __shfl_sync(0xffffffffu, uxj, from);
        uyj = __shfl_sync(0xffffffffu, uyj, from);
        uzj = __shfl_sync(0xffffffffu, uzj, from);
    }
    if (li) {
        atomicAdd(&a.ox[i], fx);
        atomicAdd(&a.oy[i], fy);
        atomicAdd(&a.oz[i], fz);
    }
    if (SYM && lj) {
        atomicAdd(&a.ox[j], gx);
        atomicAdd(&a.oy[j], gy);
        atomicAdd(&a.oz[j], gz);
    }
}

__global__ void __launch_bounds__(32 * kPairWarps) jtv_pairs64_kernel(JPair64Args a) {
    const int64_t v = (int64_t)blockIdx.x * kPairWarps + (threadIdx.x >> 5);
    for (int d = blockIdx.y; d <= a.nb / 2; d += gridDim.y) {
        int A, B, ch;
        if (!unit_blocks(v, d, a.nb, 1, A, B, ch)) return;
        if (A != B) jtv64_unit<true>(a, A, B);
        else jtv64_unit<false>(a, A, B);
    }
}

// Mixed precision.  The adjoint amplifies the error of close pairs over a rollout
// (a pair at a few softening lengths dominates J), so the pair arithmetic is FP32
// on hi/lo splits:
//   d = x_k - x_j from offsets to the block's middle particle, with the parts
// below their rounding kept where a tile comes near the block (as the direct
// sum), and
//   w = (q_j u_k,hi - q_k u_j,hi) + (q_j u_k,lo - q_k u_j,lo)
// so a small difference of two large, nearly equal adjoints keeps its digits.
// Units: coordinates in 2^-30 m (1/s^3 in metres overflows FP32), u scaled by
// a power of two from max|u|; both are exact and undone in FP64 at the end.
// The reciprocal square root is refined by one Newton step.  FP32-pipe bound:
// 45 operations per pair (39 when all charges are equal), two targets per packed
// instruction, each pair once: 16,384 particles 532 -> 217 us per launch, 4,096
// 54 -> 22 us, against the one-sided scalar kernel.  Wide plumes (kWide) keep a third
// part of their coordinates.
struct JPairArgs {
    const float4 *ph, *pl, *uh, *ul;
    const float4 *pr;  // wide plumes
    int n, nb, ct, nch;
    float e2;
    double *ox, *oy, *oz;
    const int *marks;
};

constexpr int kJR = 4, kJH = kJR / 2;  // particles (packed pairs) of the block per lane

struct JBlock {
    float2 X[kJH], Y[kJH], Z[kJH], Q[kJH], ux[kJH], uy[kJH], uz[kJH], vx[kJH], vy[kJH], vz[kJH];
    float2 fx[kJH], fy[kJH], fz[kJH];
};
struct JLow {
    float2 x[kJH][32], y[kJH][32], z[kJH][32];
    float2 rx[kJH][32], ry[kJH][32], rz[kJH][32];
};
// the travelling particle: negated coordinates and what they leave out, charge, negated u (hi, lo), and its sums
struct JTravel {
    float x, y, z, mx, my, mz, kx, ky, kz;
    float q = 0.f, ux = 0.f, uy = 0.f, uz = 0.f, vx = 0.f, vy = 0.f, vz = 0.f, sx = 0.f, sy = 0.f, sz = 0.f;
};

__device__ __forceinline__ float2 dup(float v) { return make_float2(v, v); }
__device__ __forceinline__ float turn(float v) { return __shfl_sync(0xffffffffu, v, ((threadIdx.x & 31) + 1) & 31); }

template <bool UQ, bool SYM, int MODE>
__device__ __forceinline__ void jtv_tile(JBlock &b, const JLow &low, float2 E2, float min_r2, JTravel &t) {
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (int step = 0; step < 32; step++) {
        float2 jx, jy, jz;
#pragma unroll
        for (int p = 0; p < kJH; p++) {
            float2 dx = __fadd2_rn(b.X[p], dup(t.x)), dy = __fadd2_rn(b.Y[p], dup(t.y)),
                   dz = __fadd2_rn(b.Z[p], dup(t.z));
            if (MODE != kTileFar) {
                float2 ex = __fadd2_rn(low.x[p][lane], dup(t.mx)), ey = __fadd2_rn(low.y[p][lane], dup(t.my)),
                       ez = __fadd2_rn(low.z[p][lane], dup(t.mz));
                if (MODE == kTileWide) {
                    ex = __fadd2_rn(ex, __fadd2_rn(low.rx[p][lane], dup(t.kx)));
                    ey = __fadd2_rn(ey, __fadd2_rn(low.ry[p][lane], dup(t.ky)));
                    ez = __fadd2_rn(ez, __fadd2_rn(low.rz[p][lane], dup(t.kz)));
                }
                dx = __fadd2_rn(dx, ex);
                dy = __fadd2_rn(dy, ey);
                dz = __fadd2_rn(dz, ez);
            }
            float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, E2)));
            r2 = make_float2(fmaxf(r2.x, min_r2), fmaxf(r2.y, min_r2));
            float2 inv = make_float2(rsqrt_ftz(r2.x), rsqrt_ftz(r2.y));
            inv = __fmul2_rn(inv, __ffma2_rn(__fmul2_rn(__fmul2_rn(r2, dup(-0.5f)), inv), inv, dup(1.5f)));
            const float2 inv2 = __fmul2_rn(inv, inv), inv3 = __fmul2_rn(inv, inv2);
            // q_j u_k - q_k u_j (the travelling u is negated)
            auto weight = [&](float2 uh, float2 ul, float th, float tl) {
                if (UQ) return __fadd2_rn(__fadd2_rn(uh, dup(th)), __fadd2_rn(ul, dup(tl)));
                return __fadd2_rn(__ffma2_rn(b.Q[p], dup(th), __fmul2_rn(dup(t.q), uh)),
                                  __ffma2_rn(b.Q[p], dup(tl), __fmul2_rn(dup(t.q), ul)));
            };
            const float2 wx = weight(b.ux[p], b.vx[p], t.ux, t.vx), wy = weight(b.uy[p], b.vy[p], t.uy, t.vy),
                         wz = weight(b.uz[p], b.vz[p], t.uz, t.vz);
            const float2 dot = __ffma2_rn(dx, wx, __ffma2_rn(dy, wy, __fmul2_rn(dz, wz)));
            const float2 dw = __fmul2_rn(__fmul2_rn(dot, inv2), __fmul2_rn(inv3, dup(-3.0f)));
            const float2 vx = __ffma2_rn(dw, dx, __fmul2_rn(wx, inv3)), vy = __ffma2_rn(dw, dy, __fmul2_rn(wy, inv3)),
                         vz = __ffma2_rn(dw, dz, __fmul2_rn(wz, inv3));
            b.fx[p] = __fadd2_rn(b.fx[p], vx);
            b.fy[p] = __fadd2_rn(b.fy[p], vy);
            b.fz[p] = __fadd2_rn(b.fz[p], vz);
            if (SYM) {
                jx = p == 0 ? vx : __fadd2_rn(jx, vx);
                jy = p == 0 ? vy : __fadd2_rn(jy, vy);
                jz = p == 0 ? vz : __fadd2_rn(jz, vz);
            }
        }
        t.x = turn(t.x);
        t.y = turn(t.y);
        t.z = turn(t.z);
        if (MODE != kTileFar) {
            t.mx = turn(t.mx);
            t.my = turn(t.my);
            t.mz = turn(t.mz);
        }
        if (MODE == kTileWide) {
            t.kx = turn(t.kx);
            t.ky = turn(t.ky);
            t.kz = turn(t.kz);
        }
        if (!UQ) t.q = turn(t.q);
        t.ux = turn(t.ux);
        t.uy = turn(t.uy);
        t.uz = turn(t.uz);
        t.vx = turn(t.vx);
        t.vy = turn(t.vy);
        t.vz = turn(t.vz);
        if (SYM) {
            t.sx = turn(t.sx - (jx.x + jx.y));
            t.sy = turn(t.sy - (jy.x + jy.y));
            t.sz = turn(t.sz - (jz.x + jz.y));
        }
    }
}

template <bool UQ, bool SYM, bool WIDE>
__device__ __forceinline__ void jtv_unit(const JPairArgs &a, JLow &low, int A, int B, int k0, int k1) {
    const int lane = threadIdx.x & 31;
    const float sc = (float)kLen;
    const int i0 = A * 32 * kJR, io = min(i0 + 16 * kJR, a.n - 1);
    const float4 oh = a.ph[io], ol = a.pl[io];
    Parts ox{oh.x, ol.x}, oy{oh.y, ol.y}, oz{oh.z, ol.z};
    // particle i's coordinates from the block's origin, in 2^-30 m
    auto coordinates = [&](int i, const float4 &h, Parts &x, Parts &y, Parts &z) {
        const float4 l = a.pl[i], r = WIDE ? a.pr[i] : make_float4(0.f, 0.f, 0.f, 0.f);
        x = parts_diff<WIDE>(Parts{h.x, l.x, r.x}, ox);
        y = parts_diff<WIDE>(Parts{h.y, l.y, r.y}, oy);
        z = parts_diff<WIDE>(Parts{h.z, l.z, r.z}, oz);
        x = Parts{x.v * sc, x.low * sc, x.rest * sc};
        y = Parts{y.v * sc, y.low * sc, y.rest * sc};
        z = Parts{z.v * sc, z.low * sc, z.rest * sc};
    };
    JBlock b;
    float ext = 0.f;
    __syncwarp();  // the previous unit's reads of `low`
    if (WIDE) {
        const float4 r = a.pr[io];
        ox.rest = r.x;
        oy.rest = r.y;
        oz.rest = r.z;
    }
#pragma unroll
    for (int p = 0; p < kJH; p++) {
        Parts x[2], y[2], z[2];
        float c[2][7];  // charge, u (hi, lo)
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int i = i0 + 32 * (2 * p + u) + lane;
#pragma unroll
            for (int e = 0; e < 7; e++) c[u][e] = 0.f;
            x[u].v = -kFar;
            if (i < a.n) {
                const float4 h = a.ph[i], uh = a.uh[i], ul = a.ul[i];
                coordinates(i, h, x[u], y[u], z[u]);
                c[u][0] = h.w;
                c[u][1] = uh.x;
                c[u][2] = uh.y;
                c[u][3] = uh.z;
                c[u][4] = ul.x;
                c[u][5] = ul.y;
                c[u][6] = ul.z;
                ext = fmaxf(ext, fmaxf(fabsf(x[u].v), fmaxf(fabsf(y[u].v), fabsf(z[u].v))));
            }
        }
        auto both = [&](int e) { return make_float2(c[0][e], c[1][e]); };
        b.X[p] = make_float2(x[0].v, x[1].v);
        b.Y[p] = make_float2(y[0].v, y[1].v);
        b.Z[p] = make_float2(z[0].v, z[1].v);
        low.x[p][lane] = make_float2(x[0].low, x[1].low);
        low.y[p][lane] = make_float2(y[0].low, y[1].low);
        low.z[p][lane] = make_float2(z[0].low, z[1].low);
        if (WIDE) {
            low.rx[p][lane] = make_float2(x[0].rest, x[1].rest);
            low.ry[p][lane] = make_float2(y[0].rest, y[1].rest);
            low.rz[p][lane] = make_float2(z[0].rest, z[1].rest);
        }
        b.Q[p] = both(0);
        b.ux[p] = both(1);
        b.uy[p] = both(2);
        b.uz[p] = both(3);
        b.vx[p] = both(4);
        b.vy[p] = both(5);
        b.vz[p] = both(6);
        b.fx[p] = b.fy[p] = b.fz[p] = make_float2(0.f, 0.f);
    }
    __syncwarp();
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ext = fmaxf(ext, __shfl_xor_sync(0xffffffffu, ext, o));
    const float q0 = UQ ? oh.w : 1.f;
    const float2 E2 = dup(a.e2);
    const float min_r2 = kMinR2 * sc * sc;
    for (int k = k0; k < k1; k++) {
        const int j = B * 32 * kJR + 32 * k + lane;
        JTravel t;
        Parts x{kFar}, y, z;
        if (j < a.n) {
            const float4 h = a.ph[j], uh = a.uh[j], ul = a.ul[j];
            coordinates(j, h, x, y, z);
            t.q = h.w;
            t.ux = -uh.x;
            t.uy = -uh.y;
            t.uz = -uh.z;
            t.vx = -ul.x;
            t.vy = -ul.y;
            t.vz = -ul.z;
        }
        const bool near = j < a.n && fmaxf(fabsf(x.v), fmaxf(fabsf(y.v), fabsf(z.v))) <= 2.f * ext;
        t.x = -x.v;
        t.y = -y.v;
        t.z = -z.v;
        t.mx = -x.low;
        t.my = -y.low;
        t.mz = -z.low;
        t.kx = -x.rest;
        t.ky = -y.rest;
        t.kz = -z.rest;
        if (!SYM || __any_sync(0xffffffffu, near)) {
            jtv_tile<UQ, SYM, WIDE ? kTileWide : kTileNear>(b, low, E2, min_r2, t);
        } else {
            jtv_tile<UQ, SYM, kTileFar>(b, low, E2, min_r2, t);
        }
        if (SYM && j < a.n) {
            atomicAdd(&a.ox[j], widen(t.sx * q0));
            atomicAdd(&a.oy[j], widen(t.sy * q0));
            atomicAdd(&a.oz[j], widen(t.sz * q0));
        }
    }
#pragma unroll
    for (int r = 0; r < kJR; r++) {
        const int i = i0 + 32 * r + lane;
        if (i >= a.n) continue;
        atomicAdd(&a.ox[i], widen((r & 1 ? b.fx[r / 2].y : b.fx[r / 2].x) * q0));
        atomicAdd(&a.oy[i], widen((r & 1 ? b.fy[r / 2].y : b.fy[r / 2].x) * q0));
        atomicAdd(&a.oz[i], widen((r & 1 ? b.fz[r / 2].y : b.fz[r / 2].x) * q0));
    }
}

// all units of a warp of a wide plume, with any charges (out of line, as the direct sum's:
// 16,384 particles 211 without it, 217 us so, 229 in line)
__device__ __noinline__ void jtv_wide(JPairArgs a, JLow &low, int64_t v) {
    for (int d = blockIdx.y; d <= a.nb / 2; d += gridDim.y) {
        int A, B, ch;
        if (!unit_blocks(v, d, a.nb, a.nch, A, B, ch)) return;
        const int k0 = ch * a.ct, k1 = min(k0 + a.ct, kJR);
        if (A != B) jtv_unit<false, true, true>(a, low, A, B, k0, k1);
        else jtv_unit<false, false, true>(a, low, A, B, k0, k1);
    }
}

__global__ void __launch_bounds__(32 * kPairWarps, 3) jtv_pairs_kernel(JPairArgs a) {
    __shared__ JLow lows[kPairWarps];
    JLow &low = lows[threadIdx.x >> 5];
    const int64_t v = (int64_t)blockIdx.x * kPairWarps + (threadIdx.x >> 5);
    if (a.marks[1] != 0) {
        jtv_wide(a, low, v);
        return;
    }
    const bool differ = a.marks[0] != 0;
    for (int d = blockIdx.y; d <= a.nb / 2; d += gridDim.y) {
        int A, B, ch;
        if (!unit_blocks(v, d, a.nb, a.nch, A, B, ch)) return;
        const int k0 = ch * a.ct, k1 = min(k0 + a.ct, kJR);
        if (differ) {
            if (A != B) jtv_unit<false, true, false>(a, low, A, B, k0, k1);
            else jtv_unit<false, false, false>(a, low, A, B, k0, k1);
        } else {
            if (A != B) jtv_unit<true, true, false>(a, low, A, B, k0, k1);
            else jtv_unit<true, false, false>(a, low, A, B, k0, k1);
        }
    }
}

__global__ void deinterleave(const double *__restrict__ a3, int64_t n, double *__restrict__ x,
                             double *__restrict__ y, double *__restrict__ z) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    x[i] = a3[3 * i];
    y[i] = a3[3 * i + 1];
    z[i] = a3[3 * i + 2];
}

__global__ void interleave(const double *__restrict__ x, const double *__restrict__ y,
                           const double *__restrict__ z, int64_t n, double *__restrict__ a3) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    a3[3 * i] = x[i];
    a3[3 * i + 1] = y[i];
    a3[3 * i + 2] = z[i];
}

int grid_of(int64_t n) { return (int)((n + 255) / 256 > 0 ? (n + 255) / 256 : 1); }
int stream_grid(int64_t n) {
    const int64_t b = (n + 255) / 256;
    return (int)(b < 1 ? 1 : (b > 16 * device_sms() ? 16 * device_sms() : b));
}

struct SixArrays {
    double *a[6];
};
// x, y, z, vx, vy, vz to (to = 1) or from a checkpoint of 6 n
__global__ void copy_state_kernel(SixArrays st, double *__restrict__ ck, int64_t n, int to) {
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < 6 * n; t += (int64_t)gridDim.x * blockDim.x) {
        const int k = (int)(t / n);
        double *p = st.a[k] + (t - k * n);
        if (to) ck[t] = *p;
        else *p = ck[t];
    }
}

sv_status copy_state(sv_ctx *c, double *ck, bool to) {
    if (c->n == 0) return SV_OK;
    copy_state_kernel<<<stream_grid(6 * c->n), 256, 0, c->stream>>>(
        SixArrays{{c->x, c->y, c->z, c->vx, c->vy, c->vz}}, ck, c->n, to ? 1 : 0);
    SV_LAUNCHED(c);
    return SV_OK;
}

// the 4 n + 2 doubles behind the adjoints, on a 16-byte boundary
double *scratch(const Adj &A) { return A.lam + 9 * A.n + (A.n & 1); }

// One reverse step that starts at ts, from its mid positions xh: the adjoints
// (lx, lv) of the step's end become those of its start.
sv_status reverse_step(sv_ctx *c, const double *xh, double ts) {
    Adj &A = *c->adj;
    const int64_t nn = A.n;
    double *lx = A.lam, *lv = lx + 3 * nn, *la = lv + 3 * nn;
    unsigned long long *umax = reinterpret_cast<unsigned long long *>(A.lE + 3);
    SV_CK(c, cudaMemsetAsync(umax, 0, sizeof(*umax), c->stream));
    adj_prep<<<stream_grid(nn), 256, 0, c->stream>>>(PrepArgs{xh, c->x, c->y, c->z, c->wstatus, lx, lv, la, c->qom,
                                                              c->t_inj, c->status, nn, ts, A.dt, c->P.e_over_amu,
                                                              c->P.k_const, A.lE, umax});
    SV_LAUNCHED(c);
    // the particles of the step's window in Morton order (a small window: sources first)
    const bool fp64 = c->P.precision == SV_PREC_FP64;
    c->fstatus = c->wstatus;
    c->S.want.zero = true;
    c->S.want.hilo = c->S.want.rest = !fp64;
    c->S.want.any_order = nn <= kAnyOrderMax;
    const sv_status st = sort_state(c, 0, nn);
    c->fstatus = nullptr;
    SV_TRY(st);
    Sorted &S = c->S;
    const int n = (int)S.n;
    double *u = scratch(A);
    float4 *uh = reinterpret_cast<float4 *>(u), *ul = uh + nn;
    adj_gather_u<<<grid_of(n), 256, 0, c->stream>>>(S.idx, n, S.qm, la, A.lE + 3, fp64 ? u : nullptr, uh, ul);
    SV_LAUNCHED(c);
    if (fp64) {
        const JPair64Args a{S.x, S.y, S.z, u, S.q, n, div_up(n, 32), c->P.softening2, S.ax, S.ay, S.az};
        jtv_pairs64_kernel<<<pair_grid(a.nb, 1), 32 * kPairWarps, 0, c->stream>>>(a);
    } else {
        JPairArgs a{S.ph, S.pl, uh, ul, S.pr, n, div_up(n, 32 * kJR), 0, 0, (float)(c->P.softening2 * kLen * kLen),
                    S.ax, S.ay, S.az, reinterpret_cast<const int *>(S.root + 14)};
        // about 16 units per SM sub-partition
        const int64_t tiles = (int64_t)a.nb * (a.nb + 1) / 2 * kJR;
        a.ct = (int)std::max<int64_t>(1, std::min<int64_t>({kMaxTiles, kJR, tiles / (64 * (int64_t)device_sms())}));
        a.nch = div_up(kJR, a.ct);
        jtv_pairs_kernel<<<pair_grid(a.nb, a.nch), 32 * kPairWarps, 0, c->stream>>>(a);
    }
    SV_LAUNCHED(c);
    adj_post<<<grid_of(n), 256, 0, c->stream>>>(S.idx, n, S.ax, S.ay, S.az, fp64 ? 0 : 1, umax, lx, lv, c->status,
                                                c->t_inj, ts, A.dt);
    SV_LAUNCHED(c);
    return SV_OK;
}

}  // namespace

void adjoint_state_changed(sv_ctx *c) {
    if (c->adj) c->adj->xh_seg = -1;
}

void adjoint_free(sv_ctx *c) {
    if (!c->adj) return;
    Adj &A = *c->adj;
    cudaFree(A.ck);
    cudaFree(A.xh);
    cudaFree(A.lam);
    cudaFree(A.fin);
    cudaFree(A.lE);
    delete c->adj;
    c->adj = nullptr;
}

}  // namespace sv

using namespace sv;

extern "C" sv_status sv_adjoint_forward(sv_ctx *c, int32_t nsteps, double dt, double t0, int32_t checkpoint_every) {
    if (!c) return SV_ERR_INVALID;
    if (!c->have_state) return set_error(c, SV_ERR_STATE, "no state uploaded");
    if (nsteps < 0 || !(dt > 0.0) || checkpoint_every < 1)
        return set_error(c, SV_ERR_INVALID, "nsteps >= 0, dt > 0, checkpoint_every >= 1 required");
    if (c->batch) return set_error(c, SV_ERR_UNSUPPORTED, "the adjoint runs on single-plume contexts");
    if (c->P.method != SV_METHOD_DIRECT || c->P.symmetry != SV_SYM_NONE)
        return set_error(c, SV_ERR_UNSUPPORTED, "the adjoint covers the direct sum without symmetry images");
    if (c->B.crash != SV_CRASH_NONE || c->B.bc != SV_BC_NONE || c->B.fold)
        return set_error(c, SV_ERR_UNSUPPORTED, "the adjoint covers drifts without crash, boundary or folding steps");
    if (c->sub.on) return set_error(c, SV_ERR_UNSUPPORTED, "the adjoint covers the single-rate leapfrog");
    if (c->en.on) return set_error(c, SV_ERR_UNSUPPORTED, "the adjoint runs without the energy bookkeeping");
    if (c->field.nt > 0)
        return set_error(c, SV_ERR_UNSUPPORTED, "the adjoint covers the uniform field only (no emitter field map)");
    SV_CK(c, cudaSetDevice(c->device));
    if (!c->adj) c->adj = new Adj();
    Adj &A = *c->adj;
    const int64_t n = c->n;
    const int nck = (nsteps + checkpoint_every - 1) / checkpoint_every + 1;
    const int seg = checkpoint_every < nsteps ? checkpoint_every : (nsteps > 0 ? nsteps : 1);
    if (A.cap < n || A.nck < nck || A.seg_cap < seg) {
        cudaFree(A.ck); cudaFree(A.xh); cudaFree(A.lam); cudaFree(A.fin); cudaFree(A.lE);
        A.ck = A.xh = A.lam = A.fin = A.lE = nullptr;
        const int64_t cap = n > 1 ? n : 1;
        SV_CK(c, cudaMalloc(&A.ck, sizeof(double) * 6 * cap * nck));
        SV_CK(c, cudaMalloc(&A.xh, sizeof(double) * 3 * cap * seg));
        SV_CK(c, cudaMalloc(&A.lam, sizeof(double) * (13 * cap + 2)));
        SV_CK(c, cudaMalloc(&A.fin, sizeof(double) * 6 * cap));
        SV_CK(c, cudaMalloc(&A.lE, sizeof(double) * 4));  // lE[3]: max |u| of a step
        A.cap = cap;
        A.nck = nck;
        A.seg_cap = seg;
    }
    A.n = n;
    A.nsteps = nsteps;
    A.every = checkpoint_every;
    A.dt = dt;
    A.t0 = t0;
    A.xh_seg = -1;
    const int last = nsteps > 0 ? (nsteps - 1) / checkpoint_every : 0;
    for (int s = 0; s < nsteps; s++) {
        const int k = s / checkpoint_every;
        if (s % checkpoint_every == 0) SV_TRY(copy_state(c, A.ck + (size_t)k * 6 * n, true));
        // the last segment's mid positions serve the backward pass as they are
        SV_TRY(leapfrog_step(c, t0 + dt * s, dt, k == last ? A.xh + (size_t)(s - k * checkpoint_every) * 3 * n : nullptr));
    }
    if (nsteps > 0) A.xh_seg = last;
    A.forward_done = true;
    return SV_OK;
}

extern "C" sv_status sv_adjoint_backward(sv_ctx *c, const double *dl_dx3, const double *dl_dv3, double *dl_dx0,
                                         double *dl_dv0, double *dl_defield) {
    if (!c || !dl_dx3 || !dl_dv3) return SV_ERR_INVALID;
    if (!c->adj || !c->adj->forward_done) return set_error(c, SV_ERR_STATE, "sv_adjoint_forward must run first");
    SV_CK(c, cudaSetDevice(c->device));
    Adj &A = *c->adj;
    const int64_t n = A.n;
    if (n != c->n) return set_error(c, SV_ERR_STATE, "state changed since sv_adjoint_forward");
    double *lx = A.lam, *ly = lx + n, *lz = ly + n, *lvx = lz + n, *lvy = lvx + n, *lvz = lvy + n;
    // final adjoints from the caller (host, 3n interleaved); staging behind the adjoints
    double *tmp = scratch(A);
    SV_CK(c, cudaMemcpyAsync(tmp, dl_dx3, sizeof(double) * 3 * n, cudaMemcpyHostToDevice, c->stream));
    deinterleave<<<grid_of(n), 256, 0, c->stream>>>(tmp, n, lx, ly, lz);
    SV_LAUNCHED(c);
    SV_CK(c, cudaMemcpyAsync(tmp, dl_dv3, sizeof(double) * 3 * n, cudaMemcpyHostToDevice, c->stream));
    deinterleave<<<grid_of(n), 256, 0, c->stream>>>(tmp, n, lvx, lvy, lvz);
    SV_LAUNCHED(c);
    SV_CK(c, cudaMemsetAsync(A.lE, 0, sizeof(double) * 3, c->stream));
    SV_TRY(copy_state(c, A.fin, true));
    const double dt = A.dt;
    for (int k = (A.nsteps - 1) / A.every; k >= 0 && A.nsteps > 0; k--) {
        const int s0 = k * A.every;
        const int s1 = s0 + A.every < A.nsteps ? s0 + A.every : A.nsteps;
        // recompute the segment from its checkpoint, keeping every x_h, unless
        // they are at hand
        if (A.xh_seg != k || c->field.nt > 0) {
            A.xh_seg = -1;
            SV_TRY(copy_state(c, A.ck + (size_t)k * 6 * n, false));
            for (int s = s0; s < s1; s++)
                SV_TRY(leapfrog_step(c, A.t0 + dt * s, dt, A.xh + (size_t)(s - s0) * 3 * n));
            A.xh_seg = k;
        }
        for (int s = s1 - 1; s >= s0; s--)
            SV_TRY(reverse_step(c, A.xh + (size_t)(s - s0) * 3 * n, A.t0 + dt * s));
    }
    SV_TRY(copy_state(c, A.fin, false));
    if (dl_dx0) {
        interleave<<<grid_of(n), 256, 0, c->stream>>>(lx, ly, lz, n, tmp);
        SV_LAUNCHED(c);
        SV_CK(c, cudaMemcpyAsync(dl_dx0, tmp, sizeof(double) * 3 * n, cudaMemcpyDeviceToHost, c->stream));
        SV_CK(c, cudaStreamSynchronize(c->stream));
    }
    if (dl_dv0) {
        interleave<<<grid_of(n), 256, 0, c->stream>>>(lvx, lvy, lvz, n, tmp);
        SV_LAUNCHED(c);
        SV_CK(c, cudaMemcpyAsync(dl_dv0, tmp, sizeof(double) * 3 * n, cudaMemcpyDeviceToHost, c->stream));
        SV_CK(c, cudaStreamSynchronize(c->stream));
    }
    if (dl_defield) {
        SV_CK(c, cudaMemcpyAsync(c->h_scalar, A.lE, sizeof(double) * 3, cudaMemcpyDeviceToHost, c->stream));
        SV_CK(c, cudaStreamSynchronize(c->stream));
        for (int d = 0; d < 3; d++) dl_defield[d] = c->h_scalar[d];
    }
    SV_CK(c, cudaStreamSynchronize(c->stream));
    return SV_OK;
}
