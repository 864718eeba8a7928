// bh.cu -- Barnes-Hut treecode on GB300.
//
// Restates BarnesHutForceCalculation::updateAcceleration
// (barnes_hut_force_calculation.cpp:574-715): tree, cell properties
// (computeCellProperties :337-390: net charge, centre of charge weighted by
// |charge|, delta = |centre of charge - geometric centre|) and the walk of
// computeForceFromTree (:417-450) with the acceptance test
// theta * (d - delta) > l  (d = sqrt(r^2 + eps^2), l = cell side, :435) and the
// monopole force q (x - c) / d^3 (:399-408); plus the rotational
// (barnes_hut_force_calculation_rotational.cpp:28-135: target rotated into
// each quadrant, force rotated back, self excluded only in quadrant 0) and
// translational (barnes_hut_force_calculation_translational.cpp:200-280:
// target shifted by each image offset, self excluded only for the centre
// image) variants.
//
// GB300 design:
//   * the octree is tree.cu's level structure built down to single-particle
//     boxes; a box is a leaf of the walk when it holds <= leaf_size particles
//     (the reference stops at one particle per leaf);
//   * cell properties are reduced bottom-up in FP64 in one launch: a CTA per box
//     of a middle level takes its whole subtree, and the last one to finish the
//     levels above;
//   * node centres and particle positions are stored as FP32 (hi, lo) pairs
//     relative to the root origin, so (target - centre) is formed as
//     (t_hi - c_hi) + (t_lo - c_lo): FP64-like differences with FP32
//     arithmetic only (the walk has no FP64 instruction);
//   * the walk is warp-cooperative over batches of cells: a warp owns TPW
//     Morton-consecutive targets and keeps a stack of (cell, mask of the targets
//     that rejected its parent).  It takes up to 32 cells off the stack at a time,
//     a lane loading each (one memory latency for 32 cells), then tests them one
//     after the other (32 / TPW at a time) from shared memory with a target per
//     lane: a target that accepts adds the monopole, the others' mask goes with
//     the cell's children onto the stack, or with the particles of a leaf into a
//     direct sum.  Each target gets exactly the cells its own walk would accept.
//     The stack is bounded: near its end the warp takes one cell at a time, which
//     adds at most seven entries per level.
#include <algorithm>
#include <cfloat>

#include "pairs.cuh"
#include "tree.cuh"

namespace sv {

struct Bh {
    void *arena = nullptr;
    size_t arena_bytes = 0;
    unsigned long long *d_counts = nullptr;  // [0] accepted cells, [1] direct pairs, [2] finished subtrees
    unsigned long long *h_counts = nullptr;
    int level_hint = -1;  // deepest level of the last tree
};

namespace {

constexpr int kBhWarps = 4;

// A cell of the walk: centre hi (xyz) and net charge, centre lo (xyz) and delta =
// |centre - geometric centre|, and (first particle, particle count, first child,
// children | level << 8); cells of all levels in one array, level by level.
struct Cells {
    float4 *hi, *lo;
    int4 *link;
};

// Cell properties, level by level (reductions in FP64).
struct PropLevel {
    int nbox, first;   // boxes, and the level's first cell in Cells
    const int *start, *child0;
    const int4 *coord;
    double *Q, *U;
    double3 *coc;
};
struct PropArgs {
    int deepest, top;  // top: the level with a CTA per box
    PropLevel lv[kMortonBits + 1];
    Cells cells;
    const double *xs, *ys, *zs, *root;
    const float *qs;
    unsigned long long *done;
};

// Properties of box b of level l (computeCellProperties :337-390): from its
// particles at the deepest level, else from its children (:358-388): centre =
// sum_c coc_c |Q_c| / sum_c U_c, the geometric centre when U = 0.
__device__ __forceinline__ void props_box(const PropArgs &a, int l, int b) {
    const PropLevel &V = a.lv[l];
    const double side = a.root[3] / (double)(1ll << l);
    const int s0 = V.start[b], s1 = V.start[b + 1];
    double q = 0, u = 0, tx = 0, ty = 0, tz = 0;
    int c0 = 0, c1 = 0;
    if (l == a.deepest) {
        // four particles' loads in flight at a time (as the children below)
        for (int j = s0; j < s1; j += 4) {
            float qj[4];
            double x[4], y[4], z[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int jj = min(j + k, s1 - 1);
                qj[k] = a.qs[jj];
                x[k] = a.xs[jj];
                y[k] = a.ys[jj];
                z[k] = a.zs[jj];
            }
#pragma unroll
            for (int k = 0; k < 4; k++) {
                if (j + k >= s1) break;
                const double qd = widen(qj[k]), aq = fabs(qd);
                q += qd;
                u += aq;
                tx += aq * (x[k] - a.root[0]);
                ty += aq * (y[k] - a.root[1]);
                tz += aq * (z[k] - a.root[2]);
            }
        }
    } else {
        const PropLevel &C = a.lv[l + 1];
        c0 = V.child0[b];
        c1 = V.child0[b + 1];
        for (int c = c0; c < c1; c += 4) {
            double qc[4], uc[4], x[4], y[4], z[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int cc = min(c + k, c1 - 1);
                qc[k] = __ldcg(&C.Q[cc]);
                uc[k] = __ldcg(&C.U[cc]);
                const double *p = reinterpret_cast<const double *>(C.coc + cc);
                x[k] = __ldcg(p);
                y[k] = __ldcg(p + 1);
                z[k] = __ldcg(p + 2);
            }
#pragma unroll
            for (int k = 0; k < 4; k++) {
                if (c + k >= c1) break;
                const double w = fabs(qc[k]);
                q += qc[k];
                u += uc[k];
                tx += x[k] * w;
                ty += y[k] * w;
                tz += z[k] * w;
            }
        }
    }
    const int4 cb = V.coord[b];
    // box coordinates are below 2^21: exact in FP32
    const double gx = widen((float)cb.x + 0.5f) * side, gy = widen((float)cb.y + 0.5f) * side,
                 gz = widen((float)cb.z + 0.5f) * side;
    double cx = gx, cy = gy, cz = gz;
    if (u != 0.0) {
        // 1 / u = y^2 / (1 - e) with e = 1 - u y^2, |e| < 4e-7, to third order
        double r;
        if (u > 1e-30 && u < 1e30) {
            const double y = rsqrt_seed_f64(u), y2 = y * y, e = fma(-u, y2, 1.0);
            r = fma(y2, fma(e, e, e), y2);
        } else {
            r = 1.0 / u;
        }
        cx = tx * r;
        cy = ty * r;
        cz = tz * r;
    }
    V.Q[b] = q;
    V.U[b] = u;
    V.coc[b] = make_double3(cx, cy, cz);
    const double dx = cx - gx, dy = cy - gy, dz = cz - gz;
    const double d2 = fma(dx, dx, fma(dy, dy, dz * dz));
    // sqrt to beyond the FP32 it is stored in: d2 y (1 + (1 - d2 y^2) / 2)
    const double y = rsqrt_seed_f64(d2), dy0 = d2 * y;
    float4 h, lo;
    split_hilo_bits(cx, h.x, lo.x);
    split_hilo_bits(cy, h.y, lo.y);
    split_hilo_bits(cz, h.z, lo.z);
    h.w = (float)q;
    lo.w = (float)fma(dy0, 0.5 * fma(-dy0, y, 1.0), dy0);
    const int g = V.first + b;
    a.cells.hi[g] = h;
    a.cells.lo[g] = lo;
    a.cells.link[g] = make_int4(s0, s1 - s0, l < a.deepest ? a.lv[l + 1].first + c0 : 0, (c1 - c0) | (l << 8));
}

// One CTA per box of level `top`: the boxes of its subtree are contiguous at every
// level; deepest level first, then up to the box itself.  The last CTA to finish
// takes the levels above.  One launch for all levels, over as many SMs as the
// middle level has boxes: one launch per fine level and a single CTA for every
// level of up to 1,024 boxes took 85 us at 65,536 ions, this 67.
constexpr int kPropThreads = 128;
constexpr int kPropTop = 256;  // the middle level: the deepest of up to this many boxes
__global__ void __launch_bounds__(kPropThreads) props_kernel(PropArgs a) {
    __shared__ int lo[kMortonBits + 1], hi[kMortonBits + 1];
    __shared__ bool last;
    if (threadIdx.x == 0) {
        int x = blockIdx.x, y = x + 1;
        for (int l = a.top;; l++) {
            lo[l] = x;
            hi[l] = y;
            if (l == a.deepest) break;
            x = a.lv[l].child0[x];
            y = a.lv[l].child0[y];
        }
    }
    __syncthreads();
    for (int l = a.deepest; l >= a.top; l--) {
        for (int b = lo[l] + threadIdx.x; b < hi[l]; b += kPropThreads) props_box(a, l, b);
        __syncthreads();
    }
    if (a.top == 0) return;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(a.done, 1ull) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int l = a.top - 1; l >= 0; l--) {
        for (int b = threadIdx.x; b < a.lv[l].nbox; b += kPropThreads) props_box(a, l, b);
        __syncthreads();
    }
}

struct BhImages {
    int kind;  // 0 none, 1 rotational, 2 translational offsets
    int count;
    const double *off;
};

struct WalkArgs {
    Cells cells;
    int deepest, leaf_size;
    const float4 *ph, *pl;   // sorted particles hi (xyz, charge) and lo (xyz, 1 = target)
    const double *xs, *ys, *zs, *qm;
    int n;
    const double *root;
    float theta, eps2;
    BhImages im;
    double *ax, *ay, *az;    // stored (one image), or added into (more)
    unsigned long long *counts;
};

constexpr int kStack = 512;                      // entries per warp
constexpr int kStackTail = 7 * kMortonBits + 8;  // room that one cell at a time can need

struct WalkShared {
    uint2 stack[kStack];      // cell, targets (bit per target)
    float4 hi[32], lo[32];    // the batch's cells, or 32 particles of its opened leaves
    float side[32];
    uint32_t mask[32];
    int idx[32];              // particles: sorted slot
    int leaf_at[32];          // first particle slot of each opened leaf of the batch
    int2 leaf[32];            // its particle range
    uint32_t leaf_mask[32];
};

// 1/sqrt(x), refined by one Newton step (the hardware's approximation alone is
// off by up to two units in the last place)
__device__ __forceinline__ float rsqrt_refined(float x) {
    const float y = rsqrt_ftz(x);
    const float r = y * fmaf(-0.5f * x * y, y, 1.5f);
    return y > 0.f && y <= FLT_MAX ? r : y;  // x beyond FP32, or zero
}

// TPW targets per warp; with fewer than 32, 32 / TPW groups of lanes share the
// targets and take different cells and particles.  blockIdx.y: the symmetry image.
template <int TPW>
__global__ void __launch_bounds__(kBhWarps * 32) bh_walk_kernel(WalkArgs a) {
    constexpr int G = 32 / TPW;
    constexpr uint32_t kAll = TPW == 32 ? 0xffffffffu : (1u << TPW) - 1u;
    __shared__ float side[kMortonBits + 1];  // cell side of every level, from the root cube on the device
    __shared__ WalkShared sh_all[kBhWarps];
    if (threadIdx.x <= a.deepest) side[threadIdx.x] = (float)(a.root[3] / (double)(1ll << threadIdx.x));
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    WalkShared &sh = sh_all[wid];
    const int tl = lane % TPW, grp = lane / TPW;
    const int i = (blockIdx.x * kBhWarps + wid) * TPW + tl;
    const bool live = i < a.n && a.qm[i] != 0.0;
    const uint32_t live_mask = __ballot_sync(0xffffffffu, live) & kAll;
    if (live_mask == 0) return;
    const int ii = i < a.n ? i : a.n - 1;
    // target position in this image's frame, and the force rotation back
    const int g = blockIdx.y;
    double tx = a.xs[ii], ty = a.ys[ii], tz = a.zs[ii];
    int cb = 1, sb = 0;
    bool self_excl = true;
    if (a.im.kind == 1) {
        // quadrant g: target rotated by -g*pi/2, force rotated by +g*pi/2
        const int cf = (g == 0) ? 1 : (g == 2 ? -1 : 0);
        const int sf = (g == 1) ? -1 : (g == 3 ? 1 : 0);
        const double px = tx, py = ty;
        tx = cf * px - sf * py;
        ty = sf * px + cf * py;
        cb = cf;
        sb = -sf;
        self_excl = g == 0;
    } else if (a.im.kind == 2) {
        const double *off = a.im.off + 3 * g;
        tx -= off[0];
        ty -= off[1];
        tz -= off[2];
        self_excl = off[0] == 0.0 && off[1] == 0.0 && off[2] == 0.0;
    }
    float thx, tlx, thy, tly, thz, tlz;
    split_hilo(tx - a.root[0], thx, tlx);
    split_hilo(ty - a.root[1], thy, tly);
    split_hilo(tz - a.root[2], thz, tlz);
    const int self = self_excl ? i : -1;
    float fx = 0.f, fy = 0.f, fz = 0.f;
    unsigned n_cells = 0, n_pairs = 0;
    if (lane == 0) sh.stack[0] = make_uint2(0u, live_mask);
    int size = 1;
    __syncwarp();
    while (size > 0) {
        // as many cells as the stack has room for their children
        const int room = (kStack - kStackTail - size) / 7;
        const int nb = min(min(32, size), max(1, room));
        size -= nb;
        uint32_t rej = 0;
        int4 link = make_int4(0, 0, 0, 0);
        if (lane < nb) {
            const uint2 e = sh.stack[size + lane];
            link = a.cells.link[e.x];
            sh.hi[lane] = a.cells.hi[e.x];
            sh.lo[lane] = a.cells.lo[e.x];
            sh.side[lane] = side[link.w >> 8];
            sh.mask[lane] = e.y;
        }
        __syncwarp();
        for (int k0 = 0; k0 < nb; k0 += G) {
            const int k = G == 1 ? k0 : min(k0 + grp, nb - 1);
            const float4 h = sh.hi[k], lo = sh.lo[k];
            const bool mine = (sh.mask[k] >> tl & 1u) && (G == 1 || k0 + grp < nb);
            const float dx = (thx - h.x) + (tlx - lo.x), dy = (thy - h.y) + (tly - lo.y),
                        dz = (thz - h.z) + (tlz - lo.z);
            const float r2 = fmaf(dx, dx, fmaf(dy, dy, fmaf(dz, dz, a.eps2)));
            const float inv = rsqrt_refined(r2);
            const bool acc = mine && a.theta * (r2 * inv - lo.w) > sh.side[k];
            if (acc) {
                const float f = h.w * (inv * inv * inv);
                fx = fmaf(f, dx, fx);
                fy = fmaf(f, dy, fy);
                fz = fmaf(f, dz, fz);
                n_cells++;
            }
            const uint32_t bal = __ballot_sync(0xffffffffu, mine && !acc);
            if (lane >= k0 && lane < k0 + G) rej = (bal >> ((lane - k0) * TPW)) & kAll;
        }
        // rejected cells: an internal one's children onto the stack
        const int level = link.w >> 8;
        const bool leaf = rej != 0 && (level == a.deepest || link.y <= a.leaf_size);
        const int nch = rej != 0 && !leaf ? link.w & 0xff : 0;
        int inc = nch;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        for (int c = 0; c < nch; c++) sh.stack[size + inc - nch + c] = make_uint2((uint32_t)(link.z + c), rej);
        size += __shfl_sync(0xffffffffu, inc, 31);
        // the leaves' particles, laid end to end, 32 at a time
        const uint32_t leaves = __ballot_sync(0xffffffffu, leaf);
        if (leaves) {
            int pinc = leaf ? link.y : 0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, pinc, o);
                if (lane >= o) pinc += t;
            }
            const int total = __shfl_sync(0xffffffffu, pinc, 31), nleaf = __popc(leaves);
            if (leaf) {
                const int r = __popc(leaves & ((1u << lane) - 1u));
                sh.leaf_at[r] = pinc - link.y;
                sh.leaf[r] = make_int2(link.x, link.y);
                sh.leaf_mask[r] = rej;
            }
            __syncwarp();
            int at = 0;  // the lane's current leaf: lanes walk forward
            for (int p0 = 0; p0 < total; p0 += 32) {
                const int p = p0 + lane, np = min(32, total - p0);
                if (p < total) {
                    while (at + 1 < nleaf && sh.leaf_at[at + 1] <= p) at++;
                    const int j = sh.leaf[at].x + (p - sh.leaf_at[at]);
                    sh.hi[lane] = a.ph[j];
                    sh.lo[lane] = a.pl[j];
                    sh.idx[lane] = j;
                    sh.mask[lane] = sh.leaf_mask[at];
                }
                __syncwarp();
#pragma unroll 2
                for (int k0 = 0; k0 < np; k0 += G) {
                    const int k = G == 1 ? k0 : min(k0 + grp, np - 1);
                    if ((sh.mask[k] >> tl & 1u) && sh.idx[k] != self && (G == 1 || k0 + grp < np)) {
                        const float4 qh = sh.hi[k], ql = sh.lo[k];
                        const float ex = (thx - qh.x) + (tlx - ql.x), ey = (thy - qh.y) + (tly - ql.y),
                                    ez = (thz - qh.z) + (tlz - ql.z);
                        const float inv = rsqrt_refined(fmaf(ex, ex, fmaf(ey, ey, fmaf(ez, ez, a.eps2))));
                        const float f = qh.w * (inv * inv * inv);
                        fx = fmaf(f, ex, fx);
                        fy = fmaf(f, ey, fy);
                        fz = fmaf(f, ez, fz);
                        n_pairs++;
                    }
                }
                __syncwarp();
            }
        }
        __syncwarp();
    }
    float sx = (float)cb * fx - (float)sb * fy, sy = (float)sb * fx + (float)cb * fy, sz = fz;
#pragma unroll
    for (int o = 16; o >= TPW; o >>= 1) {
        sx += __shfl_xor_sync(0xffffffffu, sx, o);
        sy += __shfl_xor_sync(0xffffffffu, sy, o);
        sz += __shfl_xor_sync(0xffffffffu, sz, o);
    }
    if (grp == 0 && live) {
        const double c = a.qm[i];
        if (a.im.count == 1) {
            a.ax[i] = (double)sx * c;
            a.ay[i] = (double)sy * c;
            a.az[i] = (double)sz * c;
        } else {
            atomicAdd(&a.ax[i], (double)sx * c);
            atomicAdd(&a.ay[i], (double)sy * c);
            atomicAdd(&a.az[i], (double)sz * c);
        }
    }
    n_cells = __reduce_add_sync(0xffffffffu, n_cells);
    n_pairs = __reduce_add_sync(0xffffffffu, n_pairs);
    if (lane == 0) {
        atomicAdd(&a.counts[0], (unsigned long long)n_cells);
        atomicAdd(&a.counts[1], (unsigned long long)n_pairs);
    }
}

}  // namespace

sv_status bh_accel(sv_ctx *c) {
    if (c->P.precision != SV_PREC_MIXED)
        return set_error(c, SV_ERR_UNSUPPORTED, "Barnes-Hut runs in mixed precision only");
    if (!c->bh) {
        c->bh = new Bh();
        SV_CK(c, cudaMalloc(&c->bh->d_counts, 3 * sizeof(unsigned long long)));
        SV_CK(c, cudaMallocHost(&c->bh->h_counts, 2 * sizeof(unsigned long long)));
    }
    Bh &B = *c->bh;
    const int n = (int)c->S.n;
    Sorted &S = c->S;
    Tree *Tp = nullptr;
    c->S.resort = false;
    SV_TRY(tree_build(c, kDepthAllSplit, c->P.leaf_size, &Tp));
    Tree &T = *Tp;
    // the splits are exact down to the sorted levels only; a tree reaching
    // them needs the full order
    if (T.n_act > 0 && T.deepest >= S.key_levels && S.key_levels < kMortonBits) {
        c->S.resort = true;
        return SV_OK;
    }
    phase_mark(c, 2);
    phase_mark(c, 3);
    SV_CK(c, cudaMemsetAsync(B.d_counts, 0, 3 * sizeof(unsigned long long), c->stream));
    if (T.n_act == 0) {
        // no source: nothing acts on anything (the scatter writes zeros for non-targets, and targets are sources)
        SV_CK(c, cudaMemcpyAsync(B.h_counts, B.d_counts, 2 * sizeof(unsigned long long), cudaMemcpyDeviceToHost,
                                 c->stream));
        return SV_OK;
    }
    const int D = T.deepest;
    B.level_hint = D;
    // storage: cells of every level, then per level Q, U (double), coc (double3)
    auto rounded = [](size_t sz) { return (sz + 255) & ~(size_t)255; };
    size_t cells = 0, bytes = 0;
    for (int l = 0; l <= D; l++) {
        const size_t nb = T.lv[l].nbox;
        cells += nb;
        bytes += 2 * rounded(nb * sizeof(double)) + rounded(nb * sizeof(double3));
    }
    bytes += 3 * rounded(cells * sizeof(float4));
    if (B.arena_bytes < bytes) {
        cudaFree(B.arena);
        B.arena = nullptr;
        B.arena_bytes = 0;
        const size_t want = bytes + bytes / 2;  // headroom: a growing tree reallocates rarely
        SV_CK(c, cudaMalloc(&B.arena, want));
        B.arena_bytes = want;
    }
    char *p = (char *)B.arena;
    auto carve = [&](size_t sz) {
        char *r = p;
        p += rounded(sz);
        return (void *)r;
    };
    PropArgs pa{};
    pa.deepest = D;
    pa.cells.hi = (float4 *)carve(cells * sizeof(float4));
    pa.cells.lo = (float4 *)carve(cells * sizeof(float4));
    pa.cells.link = (int4 *)carve(cells * sizeof(int4));
    int first = 0;
    for (int l = 0; l <= D; l++) {
        const size_t nb = T.lv[l].nbox;
        double *Q = (double *)carve(nb * sizeof(double)), *U = (double *)carve(nb * sizeof(double));
        pa.lv[l] = PropLevel{(int)nb, first, T.lv[l].start, T.lv[l].child0, T.lv[l].coord, Q, U,
                             (double3 *)carve(nb * sizeof(double3))};
        first += (int)nb;
        if (l == 0 || nb <= kPropTop) pa.top = l;
    }
    pa.xs = S.x;
    pa.ys = S.y;
    pa.zs = S.z;
    pa.qs = S.q;
    pa.root = S.root;
    pa.done = B.d_counts + 2;
    props_kernel<<<pa.lv[pa.top].nbox, kPropThreads, 0, c->stream>>>(pa);
    SV_LAUNCHED(c);
    phase_mark(c, 4);
    phase_mark(c, 5);
    BhImages im{0, 1, nullptr};
    if (c->P.symmetry == SV_SYM_ROTATIONAL) {
        im.kind = 1;
        im.count = 4;
    } else if (c->P.symmetry == SV_SYM_TRANSLATIONAL) {
        const ImageSet *I = nullptr;
        SV_TRY(image_set(c, &I));
        im.kind = 2;
        im.count = I->count;
        im.off = I->m;
    }
    // Targets per warp: 32 from 32 such warps per SM on, 16 from 8, else 8 (more
    // warps, each walking the union of fewer targets' cells).  us per evaluation
    // with 32 / 16 / 8: 1,500 ions 230 / 191 / 168, 16,000 277 / 239 / 213, 65,536
    // 392 / 374 / 374, 300,000 751 / 777 / 827.
    // inactive sorted slots (beyond n_act) are never targets (qm = 0)
    const WalkArgs wa{pa.cells, D, c->P.leaf_size, S.ph, S.pl, S.x, S.y, S.z, S.qm, T.n_act, S.root, c->P.theta,
                      (float)c->P.softening2, im, S.ax, S.ay, S.az, B.d_counts};
    auto walk = [&](auto kernel, int tpw) {
        kernel<<<dim3(div_up(T.n_act, tpw * kBhWarps), im.count), 32 * kBhWarps, 0, c->stream>>>(wa);
    };
    const int64_t warps = (int64_t)div_up(T.n_act, 32) * im.count;
    if (warps >= 32 * (int64_t)device_sms()) walk(bh_walk_kernel<32>, 32);
    else if (warps >= 8 * (int64_t)device_sms()) walk(bh_walk_kernel<16>, 16);
    else walk(bh_walk_kernel<8>, 8);
    SV_LAUNCHED(c);
    phase_mark(c, 6);
    // the counts reach the host with the stream; bh_counts reads them
    SV_CK(c, cudaMemcpyAsync(B.h_counts, B.d_counts, 2 * sizeof(unsigned long long), cudaMemcpyDeviceToHost,
                             c->stream));
    c->stats.levels = D;
    c->stats.boxes = 0;
    for (int l = 0; l <= D; l++) c->stats.boxes += T.lv[l].nbox;
    return SV_OK;
}

void bh_sort_wants(sv_ctx *c) {
    c->S.want.hilo = true;
    c->S.want.zero = c->P.symmetry != SV_SYM_NONE;  // the images' forces are added up
}

int bh_sort_levels(const sv_ctx *c) {
    const int h = c->bh ? c->bh->level_hint : -1;
    return h >= 1 ? std::min(kMortonBits, h + 2) : kMortonBits;
}

sv_status bh_counts(sv_ctx *c, double *cells, double *pairs) {
    if (!c->bh) {
        *cells = *pairs = 0;
        return SV_OK;
    }
    SV_CK(c, cudaStreamSynchronize(c->stream));
    *cells = (double)c->bh->h_counts[0];
    *pairs = (double)c->bh->h_counts[1];
    return SV_OK;
}

void bh_free(sv_ctx *c) {
    if (!c->bh) return;
    Bh &B = *c->bh;
    cudaFree(B.arena);
    cudaFree(B.d_counts);
    cudaFreeHost(B.h_counts);
    delete c->bh;
    c->bh = nullptr;
}

}  // namespace sv
