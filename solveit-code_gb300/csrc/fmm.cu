// fmm.cu -- rotation-based fast multipole method on GB300.
//
// Restates MultipoleMethodForceCalculation::updateAccelerationNoSym
// (multipole_method_force_calculation.cpp:184-522) and its kernels
// (fmm_cpukernel.cpp: p2m_kernel :281-384, m2m_kernel :513-619, m2l_kernel
// :742-909 with rotation() :10-32, l2l_kernel :1050-1126, l2p_kernel
// :1188-1317, p2p_kernel :194-219) on the level-by-level octree of tree.cu:
//
//   P2M   leaf boxes, one warp per box, lanes over particles, then over
//         coefficients (shared-memory transpose).
//   M2M   one warp per parent, lanes over the parent's coefficients, children
//         added in turn (no mutex: one writer per parent); coarse levels in one
//         launch of one CTA.
//   lists near boxes (|offset| <= ws) and the M2L list (offset class = integer
//         offset target - source): every level in two launches; the forest's
//         per level from the parents' near lists.
//   down  one warp per box and level: L2L from the parent, then every M2L of
//         the box's list (phase, folded y-rotation, z-translation, inverse
//         rotation, inverse phase), accumulated in registers, written once.
//   L2P   leaf boxes, lanes over particles: gradient of the local expansion.
//   P2P   leaf boxes, a CTA per box or chunk of its targets; groups of
//         threads, two targets each, share the sources staged in shared memory
//         as FP32 offsets from the target box centre; FP32 partial sums of at
//         most 32 sources are accumulated with Kahan compensation.
//
// Expansions are kept in box units (coordinates divided by the box side h),
// so the M2L tables depend on the integer offset only; the softened M2L
// distance rho^2 = |offset|^2 + eps^2/h^2 follows fmm_cpukernel.cpp:832.
// ws (well-separation) 1 is the reference's interaction list
// (multipole_method_force_calculation.cpp:2021-2114); ws 2 widens the near
// field to 5x5x5 boxes, which is what brings p = 8 under 1e-5 force error.
#include <cfloat>

#include <algorithm>
#include <string>
#include <vector>

#include "fmm_tables.h"
#include "forest.cuh"
#include "m2l_tc.cuh"
#include "sv_internal.cuh"
#include "tree.cuh"

namespace sv {

constexpr int kItemClasses = 32;           // near-field work items by log2 of their estimated pairs
constexpr int kCounts = 5 + kItemClasses;  // words of Fmm::d_counts

struct Fmm {
    int p = 0, ws = 0;
    int trim = 0;  // trimmed near field (sv_params.fmm_near = 2 at ws = 2) for the next evaluation
    FmmTables H;
    int *cls_theta = nullptr;
    float2 *cls_phase = nullptr;
    float *cls_rho2 = nullptr;
    float *dmat = nullptr;
    float *zc = nullptr;
    float *nrm = nullptr;
    float *otab = nullptr;   // rotation-based M2M / L2L tables (oct_layout)
    void *arena = nullptr;
    size_t arena_bytes = 0;
    unsigned long long *d_counts = nullptr;  // [0] M2L translations, [1] P2P pairs, [2] charges differ, [3] P2P work
                                             // items, [4] finished target-flag CTAs, then per size class of
                                             // the items (ints) their number and the number placed
    unsigned long long *h_counts = nullptr;
    // caller particles followed by their source-only symmetry images
    double *ex = nullptr, *ey = nullptr, *ez = nullptr, *eq = nullptr, *em = nullptr;
    int32_t *est = nullptr;
    int64_t ecap = 0;
    int *has_tgt = nullptr;  // per box of every level: nonzero if it holds a target (leaves: how many)
    int64_t tgt_cap = 0;
    float4 *rel = nullptr;   // particle offset from its leaf box centre (FP32) + charge
    int64_t rel_cap = 0;
    double *far = nullptr;   // far-field acceleration (L2P / M2P), 3 x rel_cap, added in the scatter
    int level_hint = -1;     // leaf level of the last evaluation (the next sort orders one level more)
    // forest (batched plumes): tree and per-level arrays carved at reserve time
    Tree *ftree = nullptr;
    void *farena = nullptr;
    size_t farena_bytes = 0;
    float2 *fM[kMortonBits + 1] = {}, *fL[kMortonBits + 1] = {}, *fpart[kMortonBits + 1] = {};
    int fchunks[kMortonBits + 1] = {};
    int *fnbr[kMortonBits + 1] = {}, *fcnt[kMortonBits + 1] = {}, *ftgt[kMortonBits + 1] = {};
    int2 *flst[kMortonBits + 1] = {};
    int *ffd = nullptr, *ffd_cnt = nullptr;  // far-direct lists of the forest's leaf boxes
    float4 *frel = nullptr;
    int2 *fitems = nullptr;  // near field's work items (box, chunk), largest first
    int64_t frel_cap = 0;
    // the near field runs on its own stream beside the upward and downward passes
    cudaStream_t side = nullptr;
    cudaEvent_t ev_fork = nullptr, ev_lists = nullptr, ev_join = nullptr, ev_near[2] = {};
    cudaEvent_t ev_rel = nullptr;  // single plume: the second stream's lists, leaf offsets (F.rel) and leaf flags are written
    M2LTc tc;                // the M2L on the tensor cores (m2l_tc.cu)
};

namespace {

constexpr int kWarps = 4;  // warps per CTA in the per-box kernels

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cconj(float2 a) { return make_float2(a.x, -a.y); }
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 cscale(float2 a, float s) { return make_float2(a.x * s, a.y * s); }

__host__ __device__ constexpr int ncoef(int P) { return P * (P + 1) / 2; }
__device__ __forceinline__ int cidx(int n, int m) { return n * (n + 1) / 2 + m; }
__device__ __forceinline__ void cnm(int c, int &n, int &m) {
    n = 0;
    while ((n + 1) * (n + 2) / 2 <= c) n++;
    m = c - n * (n + 1) / 2;
}

// Regular solid harmonics R_n^m(x), m >= 0, n < P (Cartesian recurrences):
// R_m^m = (x+iy)/(2m) R_{m-1}^{m-1}; R_{m+1}^m = z R_m^m;
// R_n^m = ((2n-1) z R_{n-1}^m - r^2 R_{n-2}^m) / ((n+m)(n-m)).
template <int P>
__device__ __forceinline__ void solid_harmonics(float x, float y, float z, float2 *R) {
    const float r2 = x * x + y * y + z * z;
    R[0] = make_float2(1.f, 0.f);
#pragma unroll
    for (int m = 0; m < P; m++) {
        if (m > 0) {
            const float2 prev = R[cidx(m - 1, m - 1)];
            const float s = 1.f / (2.f * m);
            R[cidx(m, m)] = make_float2((x * prev.x - y * prev.y) * s, (x * prev.y + y * prev.x) * s);
        }
        if (m + 1 < P) R[cidx(m + 1, m)] = cscale(R[cidx(m, m)], z);
#pragma unroll
        for (int n = m + 2; n < P; n++) {
            const float a = (2.f * n - 1.f) * z, d = 1.f / ((n + m) * (n - m));
            const float2 r1 = R[cidx(n - 1, m)], r0 = R[cidx(n - 2, m)];
            R[cidx(n, m)] = make_float2((a * r1.x - r2 * r0.x) * d, (a * r1.y - r2 * r0.y) * d);
        }
    }
}

// Box count of a level: the launch bound nbox, or (forest) the device count.
__device__ __forceinline__ int level_boxes(int nbox, const int *nbd) { return nbd ? min(nbox, *nbd) : nbox; }
// Root record (origin xyz, cube side) of the plume that owns box b.
__device__ __forceinline__ const double *box_root(const double *root, const int *bpid, int b) {
    return bpid ? root + 8 * bpid[b] : root;
}
// First box and stride of the calling warp in a warp-per-box kernel.
#define SV_WARP_BOXES(W) \
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5; \
    const int nb_ = level_boxes(nbox, nbd); \
    for (int b = blockIdx.x * (W) + wid; b < nb_; b += gridDim.x * (W))

// ---------------------------------------------------------------- lists --
// Lists of one box b (coordinates cb, parent par) from its parent's near list
// pnbr: the children of each of the parent's near boxes are classified round
// by round (lanes take the parent's near slots) into the near list (|offset|
// <= WS, written when write_near) and the interaction list (M2L entries
// compacted by ballot).  trim: the trimmed near field of WS = 2, whose
// (2,2,1)- and (2,2,2)-type offsets are interaction-list entries instead
// (fmm_trimmable); the near boxes of a box always have parents at offsets in
// [-1, 1]^3 from its parent, which trimming never removes, so every pair is
// still counted once.  Returns the box's M2L count.
//
// Far-direct lists (fd non-null, the leaf level of a single tree): an
// interaction-list entry whose two boxes hold fewer than fd_thresh particles
// multiplied is cheaper as direct pairs than as an M2L translation; up to
// fd_cap of them per box go to fd (summed by the near field), the rest stay
// M2L entries.
template <int WS>
__device__ __forceinline__ int build_lists_box(int b, int4 cb, int par, const int4 *__restrict__ coord,
                                               const int *__restrict__ pnbr, const int *__restrict__ pchild0,
                                               int *__restrict__ nbr, int2 *__restrict__ m2l,
                                               int *__restrict__ m2l_cnt, int cap, int write_near, int trim,
                                               const int *__restrict__ start = nullptr, int *__restrict__ fd = nullptr,
                                               int *__restrict__ fd_cnt = nullptr, int fd_cap = 0,
                                               int fd_thresh = 0) {
    constexpr int NS1 = 2 * WS + 1, NS = NS1 * NS1 * NS1, R = 2 * WS + 1, SIDE = 2 * R + 1;
    const int lane = threadIdx.x & 31;
    const unsigned lt_mask = (1u << lane) - 1u;
    if (write_near)
        for (int s = lane; s < NS; s += 32) nbr[b * NS + s] = -1;
    __syncwarp();
    const long long nt = fd ? (long long)(start[b + 1] - start[b]) : 0;
    int cnt = 0, dcnt = 0;
    for (int s0 = 0; s0 < NS; s0 += 32) {
        const int s = s0 + lane;
        int c0 = 0, c1 = 0;
        if (s < NS) {
            const int Q = pnbr[par * NS + s];
            if (Q >= 0) {
                c0 = pchild0[Q];
                c1 = pchild0[Q + 1];
            }
        }
        for (int r = 0; r < 8; r++) {
            const int ch = c0 + r;
            bool far = false;
            int cls = 0;
            if (ch < c1) {
                const int4 cc = coord[ch];
                const int ox = cb.x - cc.x, oy = cb.y - cc.y, oz = cb.z - cc.z;
                const int am = max(abs(ox), max(abs(oy), abs(oz)));
                // a consistent tree keeps |offset| <= R; a forest level clamped to
                // its capacity may not, and its result is discarded, but the class
                // index must stay inside the tables
                if (am <= WS && !(trim && fmm_trimmable(ox, oy, oz, WS))) {
                    if (write_near) nbr[b * NS + ((ox + WS) * NS1 + (oy + WS)) * NS1 + (oz + WS)] = ch;
                } else if (am <= R) {
                    far = true;
                    cls = ((ox + R) * SIDE + (oy + R)) * SIDE + (oz + R);
                }
            }
            if (fd) {
                const bool dir = far && (long long)(start[ch + 1] - start[ch]) * nt < (long long)fd_thresh;
                const unsigned bd = __ballot_sync(0xffffffffu, dir);
                if (dir) {
                    const int pos = dcnt + __popc(bd & lt_mask);
                    if (pos < fd_cap) {
                        fd[(size_t)b * fd_cap + pos] = ch;
                        far = false;
                    }
                }
                dcnt += __popc(bd);
            }
            const unsigned bal = __ballot_sync(0xffffffffu, far);
            if (far) {
                const int pos = cnt + __popc(bal & lt_mask);
                if (pos < cap) m2l[(size_t)b * cap + pos] = make_int2(ch, cls);
            }
            cnt += __popc(bal);
            if (!__any_sync(0xffffffffu, ch + 1 < c1)) break;
        }
    }
    if (cnt > cap) cnt = cap;
    if (lane == 0) {
        m2l_cnt[b] = cnt;
        if (fd) fd_cnt[b] = dcnt < fd_cap ? dcnt : fd_cap;
    }
    return cnt;
}

// One level of a forest, one warp per box.
template <int WS>
__global__ void __launch_bounds__(kWarps * 32)
build_lists_kernel(int nbox, const int *__restrict__ nbd, const int *__restrict__ parent,
                   const int4 *__restrict__ coord, const int *__restrict__ pnbr, const int *__restrict__ pchild0,
                   int *__restrict__ nbr, int2 *__restrict__ m2l, int *__restrict__ m2l_cnt, int cap, int trim,
                   unsigned long long *__restrict__ counts, const int *__restrict__ start = nullptr,
                   int *__restrict__ fd = nullptr, int *__restrict__ fd_cnt = nullptr, int fd_cap = 0,
                   int fd_thresh = 0) {
    unsigned long long tot = 0;
    SV_WARP_BOXES(kWarps) {
    const int cnt = build_lists_box<WS>(b, coord[b], parent[b], coord, pnbr, pchild0, nbr, m2l, m2l_cnt, cap, 1,
                                        trim, start, fd, fd_cnt, fd_cap, fd_thresh);
    if (lane == 0) tot += cnt;
    }
    if ((threadIdx.x & 31) == 0 && tot) atomicAdd(&counts[0], tot);
}

// The levels of one tree for the list builders that take all levels in one
// launch: level l's boxes are global indices [first, first + nbox).
struct ListLevel {
    int nbox, first;
    const int4 *coord;
    uint64_t *code;          // box Morton codes at this level (ascending)
    int *nbr;                // near lists [nbox][NS]
    const int *parent;       // box -> parent box at level - 1
    const int *pchild0;      // the parent level's child ranges
    const int *pnbr;         // the parent level's near lists
    int2 *m2l;
    int *m2l_cnt;
    const int *start;        // particle ranges of this level's boxes
    int *fd, *fd_cnt;        // far-direct lists (the leaf level only, else null)
};
struct ListArgs {
    int nlev, total;         // levels 0 .. nlev - 1; boxes of all of them
    int fd_cap, fd_thresh;   // far-direct list capacity per box and pair threshold
    int trim;                // trimmed near field (build_lists_box)
    ListLevel lv[kMortonBits + 1];
};

__device__ __forceinline__ int list_level(const ListArgs &a, int g) {
    int l = 0;
    while (l + 1 < a.nlev && g >= a.lv[l + 1].first) l++;
    return l;
}

__device__ __forceinline__ uint64_t box_code(int x, int y, int z) {
    return morton_spread3((uint32_t)x) | (morton_spread3((uint32_t)y) << 1) | (morton_spread3((uint32_t)z) << 2);
}

// Morton code of every box of every level (a level's boxes are in ascending
// code order)
__global__ void box_codes_kernel(ListArgs a) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= a.total) return;
    const ListLevel &L = a.lv[list_level(a, g)];
    const int b = g - L.first;
    const int4 c = L.coord[b];
    L.code[b] = box_code(c.x, c.y, c.z);
}

// Near lists of every level straight from the boxes (one thread per box and
// slot): the box at target - offset, found by binary search over the level's
// codes, or -1; build_lists_box's layout, without a chain of coarser levels in
// front of it.
template <int WS>
__global__ void near_lists_kernel(ListArgs a) {
    constexpr int NS1 = 2 * WS + 1, NS = NS1 * NS1 * NS1;
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= (int64_t)a.total * NS) return;
    const int g = (int)(t / NS), s = (int)(t - (int64_t)g * NS);
    const int l = list_level(a, g);
    const ListLevel &L = a.lv[l];
    const int b = g - L.first;
    const int ox = s / (NS1 * NS1) - WS, oy = (s / NS1) % NS1 - WS, oz = s % NS1 - WS;
    const int4 cb = L.coord[b];
    const int x = cb.x - ox, y = cb.y - oy, z = cb.z - oz, side = 1 << l;
    int found = -1;
    if (x >= 0 && y >= 0 && z >= 0 && x < side && y < side && z < side && !(a.trim && fmm_trimmable(ox, oy, oz, WS))) {
        const uint64_t key = box_code(x, y, z);
        int lo = 0, hi = L.nbox - 1;
        while (lo <= hi) {
            const int mid = (lo + hi) >> 1;
            const uint64_t cm = L.code[mid];
            if (cm == key) {
                found = mid;
                break;
            }
            if (cm < key) lo = mid + 1;
            else hi = mid - 1;
        }
    }
    L.nbr[(size_t)b * NS + s] = found;
}

// Interaction lists of levels 1 .. nlev - 1, one warp per box, from the near
// lists near_lists_kernel wrote
template <int WS>
__global__ void __launch_bounds__(kWarps * 32) m2l_lists_kernel(ListArgs a, int cap,
                                                                unsigned long long *__restrict__ counts) {
    unsigned long long tot = 0;
    const int lane = threadIdx.x & 31;
    const int first = a.nlev > 1 ? a.lv[1].first : a.total;
    for (int g = first + blockIdx.x * kWarps + (int)(threadIdx.x >> 5); g < a.total; g += gridDim.x * kWarps) {
        const ListLevel &L = a.lv[list_level(a, g)];
        const int b = g - L.first;
        const int cnt = build_lists_box<WS>(b, L.coord[b], L.parent[b], L.coord, L.pnbr, L.pchild0, L.nbr, L.m2l,
                                            L.m2l_cnt, cap, 0, a.trim, L.start, L.fd, L.fd_cnt, a.fd_cap,
                                            a.fd_thresh);
        if (lane == 0) tot += cnt;
    }
    if (lane == 0 && tot) atomicAdd(&counts[0], tot);
}

// Near list of every root: the root itself only (plumes never interact).
__global__ void root_nbr_kernel(int *nbr, int ns, int nroots, const int *__restrict__ nbd) {
    const int nr = level_boxes(nroots, nbd);
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nr * ns; t += gridDim.x * blockDim.x) {
        const int b = t / ns, s = t - b * ns;
        nbr[t] = s == ns / 2 ? b : -1;
    }
}

// ------------------------------------------------------ symmetry images --
// Image g of particle i at slot g*n + i: g = 0 is the particle itself; the
// others are source-only copies (status 2) rotated by g*pi/2 about z
// (rotational variant) or shifted by offset g (translational variant, zero
// offset first).  Sources of status 1 or 2 keep being sources in every image;
// ignored particles (0, -1) stay ignored.
__global__ void expand_images_kernel(const double *__restrict__ x, const double *__restrict__ y,
                                     const double *__restrict__ z, const double *__restrict__ q,
                                     const double *__restrict__ m, const int32_t *__restrict__ st, int64_t n,
                                     int kind, int nimg, const double *__restrict__ off, double *__restrict__ ex,
                                     double *__restrict__ ey, double *__restrict__ ez, double *__restrict__ eq,
                                     double *__restrict__ em, int32_t *__restrict__ est) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= n * nimg) return;
    const int g = (int)(t / n);
    const int64_t i = t - (int64_t)g * n;
    double px = x[i], py = y[i], pz = z[i];
    if (kind == 1) {
        const double x0 = px, y0 = py;
        if (g == 1) { px = -y0; py = x0; }
        else if (g == 2) { px = -x0; py = -y0; }
        else if (g == 3) { px = y0; py = -x0; }
    } else if (kind == 2) {
        px += off[3 * g];
        py += off[3 * g + 1];
        pz += off[3 * g + 2];
    }
    ex[t] = px;
    ey[t] = py;
    ez[t] = pz;
    eq[t] = q[i];
    em[t] = m[i];
    const int32_t w = st[i];
    est[t] = g == 0 ? w : ((w == 1 || w == 2) ? 2 : w);
}

// box holds at least one target (K q/m != 0).  Forest: leaf level from particles,
// coarser levels from children, a launch each (its box counts are only known on
// the device, and its launches are cheap graph nodes)
__global__ void parent_targets_kernel(int nbox, const int *__restrict__ nbd, const int *__restrict__ child0,
                                      const int *__restrict__ cflag, int *__restrict__ flag) {
    const int nb = level_boxes(nbox, nbd);
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nb; b += gridDim.x * blockDim.x) {
        int f = 0;
        for (int c = child0[b]; c < child0[b + 1] && !f; c++) f = cflag[c];
        flag[b] = f;
    }
}

// Single tree: the levels above the leaves in one launch (the leaf flags come
// with the leaf offsets).  A CTA takes the subtree of one box of level `top`; the
// last CTA to finish takes the levels above.  (Letting every leaf climb and mark
// its ancestors had all of them write the same few flags: 184 us for 10,121
// leaves.)
struct TargetArgs {
    int L, top;
    int nbox[kMortonBits + 1];
    const int *child0[kMortonBits + 1];
    int *flag[kMortonBits + 1];
    unsigned *done;                   // zero before; CTAs that have finished
};
constexpr int kFlagThreads = 256;
constexpr int kFlagTop = 8;  // the middle level: the deepest of up to this many boxes per SM

__device__ __forceinline__ void target_flag(const TargetArgs &a, int l, int b) {
    int f = 0;
    for (int c = a.child0[l][b]; c < a.child0[l][b + 1] && !f; c++) f = __ldcg(&a.flag[l + 1][c]);
    a.flag[l][b] = f;
}

__global__ void __launch_bounds__(kFlagThreads) target_flags_kernel(TargetArgs a) {
    __shared__ int lo[kMortonBits + 1], hi[kMortonBits + 1];
    __shared__ bool last;
    if (threadIdx.x == 0) {
        int x = blockIdx.x, y = x + 1;
        for (int l = a.top;; l++) {
            lo[l] = x;
            hi[l] = y;
            if (l == a.L) break;
            x = a.child0[l][x];
            y = a.child0[l][y];
        }
    }
    __syncthreads();
    for (int l = a.L - 1; l >= a.top; l--) {
        __syncthreads();
        for (int b = lo[l] + threadIdx.x; b < hi[l]; b += kFlagThreads) target_flag(a, l, b);
    }
    if (a.top == 0) return;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(a.done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int l = a.top - 1; l >= 0; l--) {
        for (int b = threadIdx.x; b < a.nbox[l]; b += kFlagThreads) target_flag(a, l, b);
        __syncthreads();
    }
}

// ------------------------------------------------------------------ P2M --
template <int P>
constexpr int p2m_warps() { return P >= 9 ? 2 : 4; }

template <int P>
__global__ void __launch_bounds__(p2m_warps<P>() * 32)
p2m_kernel(int nbox, const int *__restrict__ nbd, const int *__restrict__ bpid, const int *__restrict__ start,
           const int4 *__restrict__ coord, const double *__restrict__ xs, const double *__restrict__ ys,
           const double *__restrict__ zs, const float *__restrict__ qs, const double *__restrict__ roots, int level,
           const float *__restrict__ nrm, float2 *__restrict__ M) {
    constexpr int NC = ncoef(P), WP = p2m_warps<P>();
    __shared__ float2 buf[WP][32][NC + 1];
    SV_WARP_BOXES(WP) {
    const double *root = box_root(roots, bpid, b);
    const double h = root[3] / (double)(1 << level);
    const int4 cb = coord[b];
    const double cx = root[0] + (cb.x + 0.5) * h, cy = root[1] + (cb.y + 0.5) * h, cz = root[2] + (cb.z + 0.5) * h;
    // the offset in FP64 (positions are large), its scaling in FP32: the FP64
    // pipe runs at 1/64 of the FP32 rate on this GPU
    const float ihf = (float)(1.0 / h);
    float2 a0 = make_float2(0.f, 0.f), a1 = make_float2(0.f, 0.f);
    const int s0 = start[b], s1 = start[b + 1];
    for (int base = s0; base < s1; base += 32) {
        const int i = base + lane;
        float2 R[NC];
        if (i < s1) {
            solid_harmonics<P>((float)(xs[i] - cx) * ihf, (float)(ys[i] - cy) * ihf, (float)(zs[i] - cz) * ihf, R);
            const float q = qs[i];
#pragma unroll
            for (int c = 0; c < NC; c++) buf[wid][lane][c] = make_float2(q * R[c].x, -q * R[c].y);
        } else {
#pragma unroll
            for (int c = 0; c < NC; c++) buf[wid][lane][c] = make_float2(0.f, 0.f);
        }
        __syncwarp();
        const int rows = min(32, s1 - base);
        for (int r = 0; r < rows && lane < NC; r++) {
            a0 = cadd(a0, buf[wid][r][lane]);
            if (lane + 32 < NC) a1 = cadd(a1, buf[wid][r][lane + 32]);
        }
        __syncwarp();
    }
    if (lane < NC) {
        int n, m;
        cnm(lane, n, m);
        M[(size_t)b * NC + lane] = cscale(a0, nrm[n * P + m]);
        if (lane + 32 < NC) {
            cnm(lane + 32, n, m);
            M[(size_t)b * NC + lane + 32] = cscale(a1, nrm[n * P + m]);
        }
    }
    __syncwarp();
    }
}

// ------------------------------------------------------------------ M2M --
// (defined after the rotation helpers below)
// ----------------------------------------------------------- downward --
// M2L of every level in one launch, then L2L level by level.  A level with few
// boxes (the coarse ones, whose lists are long) splits each box's list over
// `chunks` warps; the chunks' partial sums are kept apart and added in order by
// the L2L pass, so the result does not depend on scheduling.
struct M2LLevel {
    int nbox;             // launch bound: boxes, or the forest capacity
    int chunks;           // warps per box
    int warp0;            // first global warp of the level
    int level;
    const int *nbd;       // device box count (forest) or null
    const int *bpid;      // plume of each box (forest) or null
    const int2 *m2l;
    const int *cnt;
    const int *has_tgt;   // boxes without targets need no local expansion
    const float2 *M;      // multipoles of the level
    float2 *out;          // [box][chunk][coefficient]; with one chunk the level's local expansions
};

struct M2LArgs {
    const int *run_if;    // non-null: run only when *run_if != 0 (the tensor-core M2L overflowed its room)
    int nlev, cap, esz, osz, dsz;
    double eps2;
    const double *root;
    const int *cls_theta;
    const float2 *cls_phase;
    const float *cls_rho2;
    const float *dmat;
    const float *zc;
    M2LLevel lv[kMortonBits + 1];
};

struct L2LArgs {
    int nbox, chunks, has_parent;
    const int *nbd;
    const int *parent;
    const int4 *coord;
    const int *has_tgt;
    const float2 *Lp;     // final locals of the parent level
    const float2 *part;   // this level's M2L partials [box][chunk]
    float2 *L;            // this level's locals (may alias part when chunks == 1)
    const float *otab;    // rotation-based translation tables
};

// rows of the coefficients held in slot 1 (the EXTRA lowest coefficients)
template <int P>
__host__ __device__ constexpr int slot1_rows() {
    constexpr int NC = ncoef(P);
    if (NC <= 32) return 1;
    int n = 0;
    while ((n + 1) * (n + 2) / 2 < NC - 32) n++;
    return n + 1;
}

// Rotation / translation rows are RS = p rounded up to 4 floats (16-byte
// rows, zero padded).  In shared memory the coefficients sit in rows of SR =
// RS + 2 complex values: A[n][m] by degree (n-major) for the rotations, B[k][n]
// by order (k-major) for the z-translation; entries outside a row's range stay
// zero, so whole float4 groups can be read without masks.  The 16-byte pad
// puts the rows of up to 8 consecutive degrees in 8 different 16-byte bank
// groups, so the lanes of a quarter warp (which read rows of different
// degrees) do not conflict.  The shared z-translation table keeps rows (k, j)
// of RS floats at k * ZK + j * RS, with the order stride ZK padded by a few
// 16-byte groups (chosen by counting, per order p, the bank groups the lanes
// of each quarter warp hit).
template <int P>
__host__ __device__ constexpr int rot_rs() { return (P + 3) / 4 * 4; }
template <int P>
__host__ __device__ constexpr int sh_rs() { return rot_rs<P>() + 2; }
template <int P>
__host__ __device__ constexpr int z_ks() { return P * rot_rs<P>() + 4 * (P >= 10 ? 7 : (P <= 4 ? 0 : 3)); }

// One output (n, mp) of a folded y-rotation: real part = E row . Re(A_n),
// imaginary part = O row . Im(A_n) (the O row starts with a zero for m = 0).
// G is the number of 4-coefficient groups to visit (a compile-time bound; a
// lane stops at the groups its degree n covers).
template <int P, int G>
__device__ __forceinline__ float2 rot_row(const float *__restrict__ D, int eoff, int ooff, const float2 *A, int n,
                                          int mp) {
    constexpr int RS = rot_rs<P>();
    // group-major blocks: group q of row r at (q * rows + r) float4s from the block start
    const float4 *E = reinterpret_cast<const float4 *>(D + eoff + RS * (n * (n + 1) / 2)) + mp;
    const float4 *O = reinterpret_cast<const float4 *>(D + ooff + RS * (n * (n - 1) / 2)) + (mp > 0 ? mp - 1 : 0);
    const float4 *A4 = reinterpret_cast<const float4 *>(A + n * sh_rs<P>());
    float re = 0.f, im = 0.f;
#pragma unroll
    for (int q = 0; q < G; q++) {
        if (4 * q <= n) {
            const float4 e = E[q * (n + 1)];
            const float4 a0 = A4[2 * q], a1 = A4[2 * q + 1];
            re = fmaf(e.x, a0.x, re);
            re = fmaf(e.y, a0.z, re);
            re = fmaf(e.z, a1.x, re);
            re = fmaf(e.w, a1.z, re);
            if (mp > 0) {
                const float4 o = O[q * n];
                im = fmaf(o.x, a0.y, im);
                im = fmaf(o.y, a0.w, im);
                im = fmaf(o.z, a1.y, im);
                im = fmaf(o.w, a1.w, im);
            }
        }
    }
    return make_float2(re, im);
}

// One output (j, k) of the translation along z:
// L'_j^k = sum_{n >= k} C[k][j][n] rho^-(j+n+1) M'_n^k  (C is zero for n < k)
template <int P>
__device__ __forceinline__ float2 ztrans_row(const float *__restrict__ zc, const float2 *Bk, int j, int k,
                                             float inv_rho) {
    constexpr int RS = rot_rs<P>();
    const float4 *Z = reinterpret_cast<const float4 *>(zc + k * z_ks<P>() + j * RS);
    const float4 *B4 = reinterpret_cast<const float4 *>(Bk + k * sh_rs<P>());
    float ip = inv_rho;
#pragma unroll
    for (int q = 0; q < 2 * P - 2; q++)
        if (q < j) ip *= inv_rho;  // rho^-(j+1)
    float re = 0.f, im = 0.f;
#pragma unroll
    for (int q = 0; q < RS / 4; q++) {
        const float4 z = Z[q];
        const float4 b0 = B4[2 * q], b1 = B4[2 * q + 1];
        const float f0 = z.x * ip;
        ip *= inv_rho;
        const float f1 = z.y * ip;
        ip *= inv_rho;
        const float f2 = z.z * ip;
        ip *= inv_rho;
        const float f3 = z.w * ip;
        ip *= inv_rho;
        re = fmaf(f0, b0.x, fmaf(f1, b0.z, fmaf(f2, b1.x, fmaf(f3, b1.z, re))));
        im = fmaf(f0, b0.y, fmaf(f1, b0.w, fmaf(f2, b1.y, fmaf(f3, b1.w, im))));
    }
    return make_float2(re, im);
}

// Offsets in the octant table (same as oct_layout on the host).
template <int P>
struct OctOff {
    static constexpr int RS = rot_rs<P>(), DSZ = 2 * RS * P * P, ZSZ = P * P * RS;
    static constexpr int rot = 0, zm2m = 2 * DSZ, zl2l = zm2m + ZSZ, ph_m2m = zl2l + ZSZ, ph_l2l = ph_m2m + 16 * P,
                         th_m2m = ph_l2l + 16 * P, th_l2l = th_m2m + 8;
};

// One output (j, k) of a z-shift by a fixed distance: sum_n Z[k][j][n] B[k][n]
// (SH: the table is in shared memory)
template <int P, bool SH>
__device__ __forceinline__ float2 zshift_row(const float *__restrict__ zt, const float2 *Bk, int j, int k) {
    constexpr int RS = rot_rs<P>();
    const float4 *Z = reinterpret_cast<const float4 *>(zt + ((size_t)k * P + j) * RS);
    const float4 *B4 = reinterpret_cast<const float4 *>(Bk + k * sh_rs<P>());
    float re = 0.f, im = 0.f;
#pragma unroll
    for (int q = 0; q < RS / 4; q++) {
        const float4 z = SH ? Z[q] : __ldg(Z + q);
        const float4 b0 = B4[2 * q], b1 = B4[2 * q + 1];
        re = fmaf(z.x, b0.x, fmaf(z.y, b0.z, fmaf(z.z, b1.x, fmaf(z.w, b1.z, re))));
        im = fmaf(z.x, b0.y, fmaf(z.y, b0.w, fmaf(z.z, b1.y, fmaf(z.w, b1.w, im))));
    }
    return make_float2(re, im);
}

// Rotation-based translation of one coefficient vector (GR normalisation,
// compact layout; `in` holds the lane's slots) along an octant direction: phase e^{i m phi}, y-rotation
// that takes the direction to +z, fixed z-shift Z, back-rotation, phase
// e^{-i m phi}; the result is added into the lane's accumulators.  A and B are
// the warp's degree-major / order-major rows, zero outside (n, m <= n).
template <int P, bool SH>
__device__ __forceinline__ void oct_translate(const float2 (&in)[2], const float2 *__restrict__ ph,
                                              const float *__restrict__ D, const float *__restrict__ Z, float2 *A,
                                              float2 *B, const int *cn, const int *cm, const int *cs,
                                              const bool *has, float2 *acc) {
    constexpr int RS = rot_rs<P>(), SR = sh_rs<P>(), G0 = RS / 4, G1 = slot1_rows<P>() / 4 + 1;
    constexpr int ESZ = RS * P * (P + 1) / 2, OSZ = RS * P * (P - 1) / 2;
#pragma unroll
    for (int t = 0; t < 2; t++)
        if (has[t]) A[cn[t] * SR + cm[t]] = cmul(in[t], ph[cm[t]]);
    __syncwarp();
    if (has[0]) B[cm[0] * SR + cn[0]] = rot_row<P, G0>(D, 0, ESZ, A, cn[0], cm[0]);
    if (has[1]) B[cm[1] * SR + cn[1]] = rot_row<P, G1>(D, 0, ESZ, A, cn[1], cm[1]);
    __syncwarp();
    if (has[0]) A[cn[0] * SR + cm[0]] = zshift_row<P, SH>(Z, B, cn[0], cm[0]);
    if (has[1]) A[cn[1] * SR + cm[1]] = zshift_row<P, SH>(Z, B, cn[1], cm[1]);
    __syncwarp();
    if (has[0]) acc[0] = cadd(acc[0], cmul(rot_row<P, G0>(D, ESZ + OSZ, 2 * ESZ + OSZ, A, cn[0], cm[0]), cconj(ph[cm[0]])));
    if (has[1]) acc[1] = cadd(acc[1], cmul(rot_row<P, G1>(D, ESZ + OSZ, 2 * ESZ + OSZ, A, cn[1], cm[1]), cconj(ph[cm[1]])));
    __syncwarp();
}

// lane slots of the translation kernels: slot 0 of every lane holds one of
// the NC - EXTRA highest coefficients, slot 1 of the first EXTRA lanes one of
// the EXTRA lowest (NC > 32 at p >= 8)
template <int P>
__device__ __forceinline__ void coef_slots(int lane, int *cn, int *cm, int *cs, bool *has) {
    constexpr int NC = ncoef(P), EXTRA = NC > 32 ? NC - 32 : 0;
    cs[0] = lane + EXTRA;
    cs[1] = lane;
    cnm(min(cs[0], NC - 1), cn[0], cm[0]);
    cnm(min(cs[1], NC - 1), cn[1], cm[1]);
    has[0] = cs[0] < NC;
    has[1] = lane < EXTRA;
}

// the lane's slots of a box's coefficients; through L2 (another warp of this
// launch may have written them)
template <int P>
__device__ __forceinline__ void load_slots(const float2 *src, const int *cs, const bool *has, float2 (&v)[2]) {
#pragma unroll
    for (int t = 0; t < 2; t++) v[t] = has[t] ? __ldcg(src + cs[t]) : make_float2(0.f, 0.f);
}

// M2M of one child: its multipole translated to the parent's centre by rotation
// (O(p^3) per child instead of the O(p^4) direct R-convolution), child -> parent
// box units folded into the z-shift table, added to acc.
template <int P, bool SH>
__device__ __forceinline__ void m2m_child(int ch, const int4 *__restrict__ ccoord, const float2 *Mc, const float *otab,
                                          float2 *A, float2 *B, const int *cn, const int *cm, const int *cs,
                                          const bool *has, float2 *acc) {
    using O = OctOff<P>;
    const int4 cc = ccoord[ch];
    const int oc = (cc.x & 1) | ((cc.y & 1) << 1) | ((cc.z & 1) << 2);
    const int th = (int)otab[O::th_m2m + oc];
    float2 in[2];
    load_slots<P>(Mc + (size_t)ch * ncoef(P), cs, has, in);
    oct_translate<P, SH>(in, reinterpret_cast<const float2 *>(otab + O::ph_m2m) + oc * P,
                         otab + O::rot + th * O::DSZ, otab + O::zm2m, A, B, cn, cm, cs, has, acc);
}

// one level, one warp per parent box
template <int P>
__global__ void __launch_bounds__(kWarps * 32)
m2m_kernel(int nbox, const int *__restrict__ nbd, const int *__restrict__ child0, const int4 *__restrict__ ccoord,
           const float2 *Mc, float2 *Mp, const float *__restrict__ otab) {
    constexpr int SR = sh_rs<P>();
    __shared__ __align__(16) float2 A[kWarps][P * SR], B[kWarps][P * SR];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int t = lane; t < P * SR; t += 32) A[wid][t] = B[wid][t] = make_float2(0.f, 0.f);
    __syncwarp();
    int cn[2], cm[2], cs[2];
    bool has[2];
    coef_slots<P>(lane, cn, cm, cs, has);
    const int nb = level_boxes(nbox, nbd);
    for (int b = blockIdx.x * kWarps + wid; b < nb; b += gridDim.x * kWarps) {
        float2 acc[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        const int ch1 = child0[b + 1];
        for (int ch = child0[b]; ch < ch1; ch++)
            m2m_child<P, false>(ch, ccoord, Mc, otab, A[wid], B[wid], cn, cm, cs, has, acc);
        if (has[0]) Mp[(size_t)b * ncoef(P) + cs[0]] = acc[0];
        if (has[1]) Mp[(size_t)b * ncoef(P) + cs[1]] = acc[1];
    }
}

// The coarse levels of a single tree in one launch: one CTA, level by level with
// barriers between them, the translation tables in shared memory.  A level with
// few boxes is a chain of dependent table loads in one warp per parent, and a
// launch of its own: 20,011 ions in a column, the five levels' ten launches took
// 102 us serialised, these two and the rest 80.  M2M: a warp per child (levels whose children
// number at most kCoarseBoxes), the translated multipoles kept in `tmp` and added
// per parent in child order.
constexpr int kCoarseBoxes = 64, kCoarseWarps = 16;
struct CoarseM2M {
    int top, last;  // levels top, top - 1, ..., last
    const float *otab;
    int nbox[kMortonBits + 1];
    const int *child0[kMortonBits + 1];
    const int4 *coord[kMortonBits + 1];
    float2 *M[kMortonBits + 1], *tmp[kMortonBits + 1];
};
template <int P>
constexpr int oct_size() { return OctOff<P>::th_l2l + 8; }
// rows A and B of every warp, then the tables
template <int P>
constexpr size_t coarse_smem() {
    return (size_t)kCoarseWarps * 2 * P * sh_rs<P>() * sizeof(float2) + (oct_size<P>() + 3) / 4 * 16;
}
template <int P, typename K>
cudaError_t dyn_smem(K kernel) {
    if (coarse_smem<P>() <= 48 * 1024) return cudaSuccess;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)coarse_smem<P>());
}
// the warp's zeroed rows and the CTA's copy of the tables
template <int P>
__device__ __forceinline__ const float *coarse_setup(const float *__restrict__ otab, float2 *ab, float2 *&A, float2 *&B) {
    constexpr int SR = sh_rs<P>();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    A = ab + 2 * wid * (P * SR);
    B = A + P * SR;
    for (int t = lane; t < P * SR; t += 32) A[t] = B[t] = make_float2(0.f, 0.f);
    float *tab = reinterpret_cast<float *>(ab + 2 * kCoarseWarps * (P * SR));
    for (int t = threadIdx.x; t < oct_size<P>(); t += blockDim.x) tab[t] = otab[t];
    __syncthreads();
    return tab;
}
template <int P>
__global__ void __launch_bounds__(kCoarseWarps * 32) m2m_coarse_kernel(CoarseM2M a) {
    constexpr int NC = ncoef(P);
    extern __shared__ __align__(16) float2 ab[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    float2 *A, *B;
    const float *tab = coarse_setup<P>(a.otab, ab, A, B);
    int cn[2], cm[2], cs[2];
    bool has[2];
    coef_slots<P>(lane, cn, cm, cs, has);
    for (int l = a.top; l >= a.last; l--) {
        float2 *tmp = a.tmp[l + 1];
        for (int ch = wid; ch < a.nbox[l + 1]; ch += kCoarseWarps) {
            float2 acc[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
            m2m_child<P, true>(ch, a.coord[l + 1], a.M[l + 1], tab, A, B, cn, cm, cs, has, acc);
            if (has[0]) tmp[(size_t)ch * NC + cs[0]] = acc[0];
            if (has[1]) tmp[(size_t)ch * NC + cs[1]] = acc[1];
        }
        __syncthreads();
        for (int t = threadIdx.x; t < a.nbox[l] * NC; t += blockDim.x) {
            const int b = t / NC, k = t - b * NC;
            const int c0 = a.child0[l][b], c1 = a.child0[l][b + 1];
            float2 acc = make_float2(0.f, 0.f);
            for (int ch = c0; ch < c1; ch++) acc = cadd(acc, __ldcg(&tmp[(size_t)ch * NC + k]));
            a.M[l][t] = acc;
        }
        __syncthreads();
    }
}

template <int P>
constexpr int m2l_warps() { return P >= 10 ? 2 : 4; }
// CTAs per SM the M2L is compiled for: the most that keep its registers
// unspilled (the kernel waits on dependent loads, so resident warps hide it)
template <int P>
constexpr int m2l_min_ctas() { return P >= 10 ? 1 : (P >= 8 ? 6 : 8); }
// list entries a warp carries through one pass of the M2L loop
template <int P>
constexpr int m2l_inflight() { return 2; }

// The z-translation table (the same for every entry) is staged once per CTA
// in shared memory; the rotation rows of each entry's polar angle are read
// from global memory (L1/L2), one 16-byte row segment per lane and group.
template <int P>
__global__ void __launch_bounds__(m2l_warps<P>() * 32, m2l_min_ctas<P>()) m2l_kernel(M2LArgs a) {
    constexpr int NC = ncoef(P), RS = rot_rs<P>(), SR = sh_rs<P>(), ZK = z_ks<P>(), WP = m2l_warps<P>();
    constexpr int NU = m2l_inflight<P>();
    if (a.run_if && !*a.run_if) return;
    __shared__ __align__(16) float2 A[WP][NU][P * SR], B[WP][NU][P * SR];
    __shared__ __align__(16) float Zsh[P * ZK];
    // the table's rows (k, j), RS floats each, to k * ZK + j * RS
    for (int t = threadIdx.x; t < P * P * (RS / 4); t += blockDim.x) {
        const int row = t / (RS / 4), g = t % (RS / 4), k = row / P, j = row % P;
        reinterpret_cast<float4 *>(Zsh + k * ZK + j * RS)[g] = __ldg(reinterpret_cast<const float4 *>(a.zc) + t);
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int t = lane; t < NU * P * SR; t += 32) {
        A[wid][t / (P * SR)][t % (P * SR)] = make_float2(0.f, 0.f);
        B[wid][t / (P * SR)][t % (P * SR)] = make_float2(0.f, 0.f);
    }
    __syncthreads();
    const int gw = blockIdx.x * WP + wid;
    int li = 0;
    while (li + 1 < a.nlev && gw >= a.lv[li + 1].warp0) li++;
    const int chunks = a.lv[li].chunks;
    const int local = gw - a.lv[li].warp0;
    const int b = local / chunks, ch = local - b * chunks;
    if (b >= level_boxes(a.lv[li].nbox, a.lv[li].nbd) || !a.lv[li].has_tgt[b]) return;
    // Lane slots.  Slot 0 of every lane holds one of the NC - EXTRA highest
    // coefficients; slot 1 of the first EXTRA lanes holds one of the EXTRA
    // lowest (cheapest) coefficients, so the second pass is short.
    constexpr int EXTRA = NC > 32 ? NC - 32 : 0;
    const int c0 = lane + EXTRA, c1 = lane;
    int cn[2], cm[2];
    cnm(min(c0, NC - 1), cn[0], cm[0]);
    cnm(min(c1, NC - 1), cn[1], cm[1]);
    const int cs[2] = {c0, c1};
    const bool has[2] = {c0 < NC, lane < EXTRA};
    float2 acc[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
    const double h = box_root(a.root, a.lv[li].bpid, b)[3] / (double)(1 << a.lv[li].level);
    const float eh2 = (float)(a.eps2 / (h * h));
    const int cnt = a.lv[li].cnt[b];
    const int per = (cnt + chunks - 1) / chunks;
    const int e0 = ch * per, e1 = min(cnt, e0 + per);
    const int2 *lst = a.lv[li].m2l + (size_t)b * a.cap;
    const float2 *Ml = a.lv[li].M;
    // NU entries in flight per iteration: their loads and the warp
    // synchronisations overlap (entries past the range's end repeat the last
    // one and are not accumulated)
    constexpr int G0 = RS / 4, G1 = slot1_rows<P>() / 4 + 1;
    for (int e = e0; e < e1; e += NU) {
        int src[NU];
        const float2 *ph[NU];
        const float *D[NU];
        float inv_rho[NU];
#pragma unroll
        for (int u = 0; u < NU; u++) {
            const int2 en = lst[min(e + u, e1 - 1)];
            src[u] = en.x;
            ph[u] = a.cls_phase + (size_t)en.y * P;
            D[u] = a.dmat + (size_t)a.cls_theta[en.y] * a.dsz;
            inv_rho[u] = rsqrtf(a.cls_rho2[en.y] + eh2);
        }
        // phase e^{i m phi}, into the degree-major rows
#pragma unroll
        for (int u = 0; u < NU; u++)
#pragma unroll
            for (int t = 0; t < 2; t++)
                if (has[t]) A[wid][u][cn[t] * SR + cm[t]] = cmul(Ml[(size_t)src[u] * NC + cs[t]], ph[u][cm[t]]);
        __syncwarp();
        // forward y-rotation (folded real matrices), into the order-major rows
#pragma unroll
        for (int u = 0; u < NU; u++) {
            if (has[0]) B[wid][u][cm[0] * SR + cn[0]] = rot_row<P, G0>(D[u], 0, a.esz, &A[wid][u][0], cn[0], cm[0]);
            if (has[1]) B[wid][u][cm[1] * SR + cn[1]] = rot_row<P, G1>(D[u], 0, a.esz, &A[wid][u][0], cn[1], cm[1]);
        }
        __syncwarp();
        // translation along z: L'_j^k = sum_n C[k][j][n] rho^-(j+n+1) M'_n^k
#pragma unroll
        for (int u = 0; u < NU; u++) {
            if (has[0]) A[wid][u][cn[0] * SR + cm[0]] = ztrans_row<P>(Zsh, &B[wid][u][0], cn[0], cm[0], inv_rho[u]);
            if (has[1]) A[wid][u][cn[1] * SR + cm[1]] = ztrans_row<P>(Zsh, &B[wid][u][0], cn[1], cm[1], inv_rho[u]);
        }
        __syncwarp();
        // backward y-rotation and phase e^{-i k phi}
#pragma unroll
        for (int u = 0; u < NU; u++) {
            if (e + u >= e1) break;
            if (has[0]) {
                const float2 r =
                    rot_row<P, G0>(D[u], a.esz + a.osz, 2 * a.esz + a.osz, &A[wid][u][0], cn[0], cm[0]);
                acc[0] = cadd(acc[0], cmul(r, cconj(ph[u][cm[0]])));
            }
            if (has[1]) {
                const float2 r =
                    rot_row<P, G1>(D[u], a.esz + a.osz, 2 * a.esz + a.osz, &A[wid][u][0], cn[1], cm[1]);
                acc[1] = cadd(acc[1], cmul(r, cconj(ph[u][cm[1]])));
            }
        }
        __syncwarp();
    }
    float2 *dst = a.lv[li].out + ((size_t)b * chunks + ch) * NC;
    if (has[0]) dst[cs[0]] = acc[0];
    if (has[1]) dst[cs[1]] = acc[1];
}

// L = (sum of the level's M2L partials, in chunk order) + L2L(parent's L),
// the L2L by rotation (O(p^3)), parent -> child box units folded into the
// z-shift table
// SH: the coarse kernel (tables in shared memory, the partials summed in a.L)
template <int P, bool SH>
__device__ __forceinline__ void l2l_box(const L2LArgs &a, const float *otab, int b, float2 *A, float2 *B, const int *cn, const int *cm,
                                        const int *cs, const bool *has) {
    constexpr int NC = ncoef(P);
    using O = OctOff<P>;
    float2 acc[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
    for (int t = 0; t < 2; t++)
        if (has[t]) {
            if (SH) acc[t] = __ldcg(&a.L[(size_t)b * NC + cs[t]]);
            else
                for (int ch = 0; ch < a.chunks; ch++)
                    acc[t] = cadd(acc[t], a.part[((size_t)b * a.chunks + ch) * NC + cs[t]]);
        }
    if (a.has_parent) {
        const int4 cb = a.coord[b];
        const int oc = (cb.x & 1) | ((cb.y & 1) << 1) | ((cb.z & 1) << 2);
        const int th = (int)otab[O::th_l2l + oc];
        float2 in[2];
        load_slots<P>(a.Lp + (size_t)a.parent[b] * NC, cs, has, in);
        oct_translate<P, SH>(in, reinterpret_cast<const float2 *>(otab + O::ph_l2l) + oc * P,
                             otab + O::rot + th * O::DSZ, otab + O::zl2l, A, B, cn, cm, cs, has, acc);
    }
    if (has[0]) a.L[(size_t)b * NC + cs[0]] = acc[0];
    if (has[1]) a.L[(size_t)b * NC + cs[1]] = acc[1];
}

template <int P>
__global__ void __launch_bounds__(kWarps * 32) l2l_kernel(L2LArgs a) {
    constexpr int SR = sh_rs<P>();
    __shared__ __align__(16) float2 A[kWarps][P * SR], B[kWarps][P * SR];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int t = lane; t < P * SR; t += 32) A[wid][t] = B[wid][t] = make_float2(0.f, 0.f);
    __syncwarp();
    int cn[2], cm[2], cs[2];
    bool has[2];
    coef_slots<P>(lane, cn, cm, cs, has);
    const int nb = level_boxes(a.nbox, a.nbd);
    for (int b = blockIdx.x * kWarps + wid; b < nb; b += gridDim.x * kWarps)
        if (a.has_tgt[b]) l2l_box<P, false>(a, a.otab, b, A[wid], B[wid], cn, cm, cs, has);
}

// the coarse levels first .. last in one CTA, as m2m_coarse_kernel
struct CoarseL2L {
    int first, last;
    L2LArgs lv[kMortonBits + 1];
};
template <int P>
__global__ void __launch_bounds__(kCoarseWarps * 32) l2l_coarse_kernel(CoarseL2L a) {
    constexpr int NC = ncoef(P);
    extern __shared__ __align__(16) float2 ab[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    float2 *A, *B;
    const float *tab = coarse_setup<P>(a.lv[a.first].otab, ab, A, B);
    int cn[2], cm[2], cs[2];
    bool has[2];
    coef_slots<P>(lane, cn, cm, cs, has);
    // every level's M2L partials first (their loads depend on nothing), in chunk order
    for (int l = a.first; l <= a.last; l++) {
        const L2LArgs &v = a.lv[l];
        for (int t = threadIdx.x; t < v.nbox * NC; t += blockDim.x) {
            const int b = t / NC, k = t - b * NC;
            if (!v.has_tgt[b]) continue;
            const float2 *p = v.part + (size_t)b * v.chunks * NC + k;
            float2 acc = make_float2(0.f, 0.f);
            for (int c0 = 0; c0 < v.chunks; c0 += 8) {
                float2 x[8];
#pragma unroll
                for (int u = 0; u < 8; u++) x[u] = p[(size_t)min(c0 + u, v.chunks - 1) * NC];
#pragma unroll
                for (int u = 0; u < 8; u++)
                    if (c0 + u < v.chunks) acc = cadd(acc, x[u]);
            }
            v.L[t] = acc;
        }
    }
    __syncthreads();
    for (int l = a.first; l <= a.last; l++) {
        if (!a.lv[l].has_parent) continue;
        for (int b = wid; b < a.lv[l].nbox; b += kCoarseWarps)
            if (a.lv[l].has_tgt[b]) l2l_box<P, true>(a.lv[l], tab, b, A, B, cn, cm, cs, has);
        __syncthreads();
    }
}

// warps per box for a level of nbox boxes: enough to give every SM a few
// warps even at the coarse levels, at most 16
inline int m2l_chunks(int nbox) {
    const int want = 16 * device_sms();
    int c = nbox > 0 ? (want + nbox - 1) / nbox : 1;
    return c < 1 ? 1 : (c > 16 ? 16 : c);
}

// ------------------------------------------------------------------ L2P --
template <int P>
__global__ void __launch_bounds__(kWarps * 32)
l2p_kernel(int nbox, const int *__restrict__ nbd, const int *__restrict__ bpid, const int *__restrict__ start,
           const float4 *__restrict__ rel, const double *__restrict__ qm, const double *__restrict__ roots, int level,
           const float *__restrict__ nrm, const float2 *__restrict__ Lc, double *__restrict__ ax,
           double *__restrict__ ay, double *__restrict__ az, const int *__restrict__ has_tgt, int accumulate) {
    constexpr int NC = ncoef(P);
    __shared__ float2 lam[kWarps][NC];
    __shared__ int wait[kWarps][64];
    SV_WARP_BOXES(kWarps) {
    const double *root = box_root(roots, bpid, b);
    if (!has_tgt[b]) {
        // boxes of image copies only: no targets, zero acceleration
        if (!accumulate)
            for (int i = start[b] + lane; i < start[b + 1]; i += 32) ax[i] = ay[i] = az[i] = 0.0;
        continue;
    }
    for (int c = lane; c < NC; c += 32) {
        int n, m;
        cnm(c, n, m);
        lam[wid][c] = cscale(Lc[(size_t)b * NC + c], nrm[n * P + m]);
    }
    __syncwarp();
    // Positions relative to the leaf box centre come from box_relative_kernel
    // (FP32, metres); the per-particle work stays on the FP32 pipe, the FP64
    // pipe (1/64 of its rate on this GPU) sees only the stores' conversions.
    const double h = root[3] / (double)(1 << level);
    const float ihf = (float)(1.0 / h), mih2 = (float)(-1.0 / (h * h));
    // Rounds of 32 particles; where the box holds more than targets (image copies), of
    // 32 targets gathered first.
    const int s1 = start[b + 1];
    const bool some = has_tgt[b] < s1 - start[b];
    int have = 0;
    for (int next = start[b];;) {
        int i = next + lane;
        bool live = i < s1;
        if (some) {
            while (have < 32 && next < s1) {
                const int k = next + lane;
                const bool f = k < s1 && qm[k] != 0.0;
                const unsigned bal = __ballot_sync(0xffffffffu, f);
                if (f) wait[wid][have + __popc(bal & ((1u << lane) - 1u))] = k;
                have += __popc(bal);
                next += 32;
                __syncwarp();
            }
            if (have == 0) break;
            live = lane < have;
            i = wait[wid][lane];
            const int left = lane + 32 < have ? wait[wid][lane + 32] : 0;
            __syncwarp();
            wait[wid][lane] = left;
            have = max(have - 32, 0);
            __syncwarp();
        } else {
            if (next >= s1) break;
            next += 32;
        }
        if (!live) continue;
        float2 R[ncoef(P - 1) > 0 ? ncoef(P - 1) : 1];
        const float4 r = rel[i];
        solid_harmonics<P - 1>(r.x * ihf, r.y * ihf, r.z * ihf, R);
        float gz = 0.f;
        float2 gm = make_float2(0.f, 0.f);
#pragma unroll
        for (int n = 1; n < P; n++) {
            const float2 *ln = &lam[wid][cidx(n, 0)];
            gz = fmaf(ln[0].x, R[cidx(n - 1, 0)].x, gz);
#pragma unroll
            for (int m = 1; m < n; m++) {
                const float2 v = cmul(ln[m], R[cidx(n - 1, m)]);
                gz = fmaf(2.f, v.x, gz);
            }
#pragma unroll
            for (int m = 1; m <= n; m++) gm = cadd(gm, cmul(ln[m], R[cidx(n - 1, m - 1)]));
#pragma unroll
            for (int t = 0; t + 1 < n; t++) gm = cadd(gm, cscale(cconj(cmul(ln[t], R[cidx(n - 1, t + 1)])), -1.f));
        }
        // a = -grad(phi) * K q / m, grad in box units / h^2 (added to the
        // near field when that ran first)
        const float f = (float)qm[i] * mih2;
        const float vx = f * gm.x, vy = -f * gm.y, vz = f * gz;
        if (accumulate) {
            ax[i] += (double)vx;
            ay[i] += (double)vy;
            az[i] += (double)vz;
        } else {
            ax[i] = (double)vx;
            ay[i] = (double)vy;
            az[i] = (double)vz;
        }
    }
    __syncwarp();
    }
}


// ----------------------------------------------------------- treecode M2P --
// The treecode mode (FmmType::treecode, m2p_kernel fmm_cpukernel.cpp:1399-1533)
// evaluates every far-field multipole directly at the target particles
// instead of translating it into local expansions.  A leaf box's particles
// receive the multipoles of the interaction lists of all its ancestors
// (levels L..2).  With M in the regular-harmonic normalisation of P2M
// (M = sum q conj(R_n^m(d)), R_n^m = r^n P_n^m e^{im phi} / (n+m)!), the
// potential is phi(x) = sum_{n,m} M_n^m S_n^m(x - c) with the irregular
// harmonics S_n^m = (n-m)! r^{-n-1} P_n^m e^{im phi}, and
//   d/dz S_n^m = -S_{n+1}^m,   (d/dx + i d/dy) S_n^m = -S_{n+1}^{m+1}.
// The softened distance r^2 + eps^2/h^2 enters the recurrences, as the
// reference softens r in its M2P and M2L.

// Irregular solid harmonics S_n^m, m >= 0, degrees 0..Q-1:
// S_0^0 = 1/r; S_m^m = (2m-1)(x+iy)/r^2 S_{m-1}^{m-1}; S_{m+1}^m = (2m+1) z/r^2 S_m^m;
// S_n^m = ((2n-1) z S_{n-1}^m - ((n-1)^2 - m^2) S_{n-2}^m) / r^2.
template <int Q>
__device__ __forceinline__ void irregular_harmonics(float x, float y, float z, float r2, float2 *S) {
    const float ir2 = 1.f / r2;
    S[0] = make_float2(rsqrtf(r2), 0.f);
#pragma unroll
    for (int m = 0; m < Q; m++) {
        if (m > 0) {
            const float2 prev = S[cidx(m - 1, m - 1)];
            const float s = (2.f * m - 1.f) * ir2;
            S[cidx(m, m)] = make_float2((x * prev.x - y * prev.y) * s, (x * prev.y + y * prev.x) * s);
        }
        if (m + 1 < Q) S[cidx(m + 1, m)] = cscale(S[cidx(m, m)], (2.f * m + 1.f) * z * ir2);
#pragma unroll
        for (int n = m + 2; n < Q; n++) {
            const float a = (2.f * n - 1.f) * z, d = (float)((n - 1) * (n - 1) - m * m);
            const float2 s1 = S[cidx(n - 1, m)], s0 = S[cidx(n - 2, m)];
            S[cidx(n, m)] = make_float2((a * s1.x - d * s0.x) * ir2, (a * s1.y - d * s0.y) * ir2);
        }
    }
}

struct TreecodeArgs {
    int L, cap, ws, nleaf;
    const int *parent[kMortonBits + 1];
    const int4 *coord[kMortonBits + 1];
    const int2 *m2l[kMortonBits + 1];
    const int *m2l_cnt[kMortonBits + 1];
    const float2 *M[kMortonBits + 1];
    const int *leaf_start;
    const int *has_tgt;
    const double *x, *y, *z, *qm;
    const double *root;
    const float *nrm;
    double eps2;
    double *ax, *ay, *az;
    int accumulate;  // 1: add to ax (the near field ran first), 0: overwrite
};

template <int P>
__global__ void __launch_bounds__(kWarps * 32) m2p_kernel(TreecodeArgs a) {
    constexpr int NC = ncoef(P), NS = ncoef(P + 1);
    __shared__ float2 Mw[kWarps][NC];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int b = blockIdx.x * kWarps + wid;
    if (b >= a.nleaf) return;
    const int s0 = a.leaf_start[b], s1 = a.leaf_start[b + 1];
    if (!a.has_tgt[b]) {
        if (!a.accumulate)
            for (int i = s0 + lane; i < s1; i += 32) a.ax[i] = a.ay[i] = a.az[i] = 0.0;
        return;
    }
    const int R = 2 * a.ws + 1, SIDE = 2 * R + 1;
    for (int tb = s0; tb < s1; tb += 32) {
        const int i = tb + lane;
        const bool valid = i < s1;
        const int ii = valid ? i : s0;
        double gx = 0.0, gy = 0.0, gz = 0.0;
        int box = b;
        for (int l = a.L; l >= 2; l--) {
            const double h = a.root[3] / (double)(1 << l);
            const int4 cb = a.coord[l][box];
            const double ih = 1.0 / h;
            const float dx0 = (float)((a.x[ii] - (a.root[0] + (cb.x + 0.5) * h)) * ih);
            const float dy0 = (float)((a.y[ii] - (a.root[1] + (cb.y + 0.5) * h)) * ih);
            const float dz0 = (float)((a.z[ii] - (a.root[2] + (cb.z + 0.5) * h)) * ih);
            const float e2 = (float)(a.eps2 * ih * ih);
            const int cnt = a.m2l_cnt[l][box];
            const int2 *lst = a.m2l[l] + (size_t)box * a.cap;
            float fx = 0.f, fy = 0.f, fz = 0.f;
            for (int e = 0; e < cnt; e++) {
                const int2 ent = lst[e];
                __syncwarp();
                for (int c = lane; c < NC; c += 32) {
                    int n, m;
                    cnm(c, n, m);
                    Mw[wid][c] = cscale(a.M[l][(size_t)ent.x * NC + c], 1.f / a.nrm[n * P + m]);
                }
                __syncwarp();
                // target ancestor minus source box, in boxes (exact)
                const int oz = ent.y % SIDE - R, oy = (ent.y / SIDE) % SIDE - R, ox = ent.y / (SIDE * SIDE) - R;
                const float dx = dx0 + (float)ox, dy = dy0 + (float)oy, dz = dz0 + (float)oz;
                float2 S[NS];
                irregular_harmonics<P + 1>(dx, dy, dz, fmaf(dx, dx, fmaf(dy, dy, fmaf(dz, dz, e2))), S);
                float2 gp = make_float2(0.f, 0.f);
                float gzz = 0.f;
#pragma unroll
                for (int n = 0; n < P; n++) {
                    const float2 *Mn = &Mw[wid][cidx(n, 0)];
                    const float2 *Sn = &S[cidx(n + 1, 0)];
                    gzz += cmul(Mn[0], Sn[0]).x;
#pragma unroll
                    for (int m = 1; m <= n; m++) gzz += 2.f * cmul(Mn[m], Sn[m]).x;
#pragma unroll
                    for (int m = 0; m <= n; m++) gp = cadd(gp, cmul(Mn[m], Sn[m + 1]));
#pragma unroll
                    for (int k = 1; k <= n; k++) gp = cadd(gp, cscale(cconj(cmul(Mn[k], Sn[k - 1])), -1.f));
                }
                fx -= gp.x;
                fy -= gp.y;
                fz -= gzz;
            }
            const double s = ih * ih;
            gx += (double)fx * s;
            gy += (double)fy * s;
            gz += (double)fz * s;
            box = a.parent[l][box];
        }
        if (valid) {
            // a = -K q/m grad(phi)
            const double c = a.qm[i];
            if (a.accumulate) {
                a.ax[i] += -c * gx;
                a.ay[i] += -c * gy;
                a.az[i] += -c * gz;
            } else {
                a.ax[i] = -c * gx;
                a.ay[i] = -c * gy;
                a.az[i] = -c * gz;
            }
        }
    }
}

// ------------------------------------------------------------------ P2P --
// Each particle once as an FP32 offset from the centre of its own leaf box
// (one FP64 subtraction per particle) with its charge: the P2P kernel then
// forms source offsets from the target box centre as offset + k*h in FP32.
// A charge other than qs[0] sets *mixed (zeroed beforehand), which keeps the
// P2P kernel on its per-source charge path.  With flag, the box's number of targets.
__global__ void __launch_bounds__(kWarps * 32)
box_relative_kernel(int nbox, const int *__restrict__ nbd, const int *__restrict__ bpid,
                    const int *__restrict__ start, const int4 *__restrict__ coord, const double *__restrict__ xs,
                    const double *__restrict__ ys, const double *__restrict__ zs, const float *__restrict__ qs,
                    const double *__restrict__ roots, int level, float4 *__restrict__ rel,
                    unsigned long long *__restrict__ mixed, const double *__restrict__ qm = nullptr,
                    int *__restrict__ flag = nullptr) {
    const float q0 = qs[0];
    bool diff = false;
    SV_WARP_BOXES(kWarps) {
    const double *root = box_root(roots, bpid, b);
    const double h = root[3] / (double)(1 << level);
    const int4 cb = coord[b];
    const double cx = root[0] + (cb.x + 0.5) * h, cy = root[1] + (cb.y + 0.5) * h, cz = root[2] + (cb.z + 0.5) * h;
    int tgt = 0;
    for (int j = start[b] + lane; j < start[b + 1]; j += 32) {
        const float q = qs[j];
        diff |= q != q0;
        rel[j] = make_float4((float)(xs[j] - cx), (float)(ys[j] - cy), (float)(zs[j] - cz), q);
        if (flag) tgt += qm[j] != 0.0;
    }
    if (flag) {
        tgt = __reduce_add_sync(0xffffffffu, tgt);
        if (lane == 0) flag[b] = tgt;
    }
    }
    if (__any_sync(0xffffffffu, diff) && (threadIdx.x & 31) == 0) *mixed = 1ull;
}

// 16-byte asynchronous copy global -> shared (LDGSTS): the data lands without
// passing through registers; the issuing thread sees it after cp_async_wait_all.
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// s += v with Kahan compensation e (the running sum is s - e)
__device__ __forceinline__ void kahan_add(float &s, float &e, float v) {
    const float y = v - e, t = s + y;
    e = (t - s) - y;
    s = t;
}

// Near field, one CTA per work item (a leaf box, or a share of its target
// chunks).  The box's non-empty near boxes, then its far-direct boxes
// (interaction-list entries cheaper as pairs, from build_lists_box), are
// compacted into shared memory with a running count of their sources; the
// sources are then streamed kSrcTile at a time across box boundaries (each
// thread walks forward to the boxes of its staged sources), so the pair loop
// runs without per-box padding or per-box overhead.  Sources are staged as
// negated coordinates in structure-of-arrays rows, so one 64-bit load gives
// two consecutive sources and each pair operation is a packed FP32x2
// instruction (FADD2 / FFMA2 / FMUL2) over two sources; the reciprocal square
// roots stay scalar.
//
// Split: a chunk of nt <= 2 kP2PThreads targets takes h = ceil(nt / 2) threads,
// two targets each, and s = kP2PThreads / h such groups (32 at most) that share
// the staged sources run by run, so the lanes stay busy whatever the box
// holds (h s / kP2PThreads, ~0.9 on average) and a box with many targets and
// sources occupies four warps instead of one.  Up to 32 sources per group are
// summed in FP32 (16 per half of the packed pair), then added with Kahan
// compensation; the groups' sums are added in group order at the end, so the
// result does not depend on scheduling.  FP32-pipe bound: 11 FMA-pipe operations and one reciprocal
// square root per pair.
//
// The result is stored (each particle of a box with targets once; boxes
// without targets are left as they are).  CLAMP: floor r^2 at kMinR2, needed
// only when eps^2 < kMinR2 (a zero-distance pair without softening).  UQ:
// every particle of the tree carries the same charge Q (box_relative_kernel
// found no other), so the pair weight is r^-3 alone, the sums are scaled by
// the target's own charge (= Q) at the end, and padding sources sit far away
// (r^-3 underflows to zero) instead of carrying zero charge.
constexpr int kFarDirectCap = 128;  // far-direct source boxes per leaf box
constexpr int kP2PThreads = 128;
constexpr int kSrcTile = 2 * kP2PThreads;  // sources staged per round, two per thread
// source boxes a leaf box's near field can take: its near boxes and its far-direct ones
template <int WS>
constexpr int p2p_nsp() { return ((2 * WS + 1) * (2 * WS + 1) * (2 * WS + 1) + 31) / 32 * 32 + kFarDirectCap; }

template <int WS>
struct P2PShared {
    float st[2][4][kSrcTile];      // staged sources (double buffer): -x, -y, -z, charge
    float4 raw[2][kSrcTile];       // the next sources as copied (double buffer; each thread its own)
    float4 nb_off[p2p_nsp<WS>()];  // source box centre - target box centre (exact in FP32)
    int2 nb_rng[p2p_nsp<WS>()];    // (first source, running source count at the box's end)
    int scan[2][kP2PThreads / 32], nz[2][kP2PThreads / 32];  // per warp and list: sources, non-empty boxes
};

// Chunks a box's nt targets are cut into.  A chunk's time per source is that
// of staging it (~60 issue slots per 256 sources and warp) plus 44 FMA-pipe
// clocks per two sources and group step, 1 / s of them per group: c chunks cost
// c (1 + 96 / s).  The least of four successive counts is taken, from `parts`
// on (so that a tree of few boxes gives every CTA slot work) unless a chunk
// would fall below 16 targets.
__device__ __forceinline__ int p2p_chunks(int nt, int parts) {
    if (nt <= 0) return 0;
    const int c0 = max((nt + 2 * kP2PThreads - 1) / (2 * kP2PThreads), min(parts, (nt + 15) / 16));
    const int c1 = max(c0, min(c0 + 3, (nt + 7) / 8));
    int best = c0;
    float cost = FLT_MAX;
    for (int c = c0; c <= c1; c++) {
        const int h = ((nt + c - 1) / c + 1) >> 1, s = min(32, kP2PThreads / h);
        const float t = (float)c * (1.f + 96.f / (float)s);
        if (t < cost) {
            cost = t;
            best = c;
        }
    }
    return best;
}

template <int WS, bool CLAMP, bool UQ, bool SOME>
__device__ __forceinline__ void
p2p_item(P2PShared<WS> &sh, int b, int ntgt, int part, int parts, int stride, const int *__restrict__ bpid, const int *__restrict__ start,
         const int4 *__restrict__ coord, const int *__restrict__ nbr, const double *__restrict__ qm,
         const double *__restrict__ roots, int level, float eps2, double *__restrict__ ax, double *__restrict__ ay,
         double *__restrict__ az, unsigned long long *__restrict__ counts, const float4 *__restrict__ rel,
         const int *__restrict__ fd, const int *__restrict__ fd_cnt, int fd_cap) {
    constexpr int NS1 = 2 * WS + 1, NS = NS1 * NS1 * NS1;
    static_assert(NS <= kP2PThreads && kFarDirectCap <= kP2PThreads, "a list is compacted in one round");
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int t0 = start[b], nt_all = SOME ? ntgt : start[b + 1] - t0;
    const int nchunk = p2p_chunks(nt_all, parts);
    if (part >= nchunk) return;
    const float4 pad = UQ ? make_float4(1e18f, 0.f, 0.f, 0.f) : make_float4(0.f, 0.f, 0.f, 0.f);
    const float2 E2 = make_float2(eps2, eps2);
    const float hf = (float)(box_root(roots, bpid, b)[3] / (double)(1 << level));
    const int4 cb = coord[b];
    int nnz = 0, total = 0;
    // the non-empty boxes of a list (-1 entries skipped) appended with their
    // running source count and their offset: one entry per thread, scanned
    // over the CTA
    auto add_boxes = [&](const int *list, int count, int round) {
        int Q = -1, j0 = 0, cnt = 0;
        if (tid < count) {
            Q = list[tid];
            if (Q >= 0) {
                j0 = start[Q];
                cnt = start[Q + 1] - j0;
            }
        }
        const bool f = cnt > 0;
        const unsigned bal = __ballot_sync(0xffffffffu, f);
        int inc = cnt;
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        if (lane == 31) sh.scan[round][wid] = inc;
        if (lane == 0) sh.nz[round][wid] = __popc(bal);
        __syncthreads();
        int pos = nnz + __popc(bal & ((1u << lane) - 1u)), run = total + inc;
#pragma unroll
        for (int w = 0; w < kP2PThreads / 32; w++) {
            if (w < wid) {
                pos += sh.nz[round][w];
                run += sh.scan[round][w];
            }
            nnz += sh.nz[round][w];
            total += sh.scan[round][w];
        }
        if (f) {
            const int4 cq = coord[Q];
            sh.nb_rng[pos] = make_int2(j0, run);
            sh.nb_off[pos] = make_float4((float)(cq.x - cb.x) * hf, (float)(cq.y - cb.y) * hf,
                                         (float)(cq.z - cb.z) * hf, 0.f);
        }
    };
    add_boxes(nbr + (size_t)b * NS, NS, 0);
    if (fd) add_boxes(fd + (size_t)b * fd_cap, fd_cnt[b], 1);
    __syncthreads();
    const int csize = (nt_all + nchunk - 1) / nchunk;
    for (int ch = part; ch < nchunk; ch += stride) {
        const int tb = t0 + ch * csize, nt = min(csize, t0 + nt_all - tb);
        // The chunk's targets by index, where the box holds other particles too: in the copy
        // buffer that is first written after the first tile's barrier.
        int *const tix = reinterpret_cast<int *>(sh.raw[1]);
        if (SOME) {
            // targets r0 .. r0 + nt of the box: ranks counted over the CTA, 128 particles a round
            const int r0 = tb - t0;
            const int np = start[b + 1] - t0;
            for (int k0 = 0, seen = 0; k0 < np && seen < r0 + nt; k0 += kP2PThreads) {
                const int k = k0 + tid;
                const bool f = k < np && qm[t0 + k] != 0.0;
                const unsigned bal = __ballot_sync(0xffffffffu, f);
                __syncthreads();
                if (lane == 0) sh.nz[0][wid] = __popc(bal);
                __syncthreads();
                int r = seen - r0 + __popc(bal & ((1u << lane) - 1u));
#pragma unroll
                for (int w = 0; w < kP2PThreads / 32; w++) {
                    if (w < wid) r += sh.nz[0][w];
                    seen += sh.nz[0][w];
                }
                if (f && r >= 0 && r < nt) tix[r] = t0 + k;
            }
            __syncthreads();
        }
        const int h = (nt + 1) >> 1, s = min(32, kP2PThreads / h);
        // each group's run of a tile: 32 consecutive sources, fewer when more than
        // eight groups share the staging rows
        const int run = s <= 8 ? 32 : (s <= 16 ? 16 : 8), tile = s * run;
        const int grp = tid / h, lt = tid - grp * h;
        const bool active = grp < s;
        const bool vb = active && lt + h < nt;
        const int ia = SOME ? tix[active ? lt : 0] : tb + lt, ib = SOME ? tix[vb ? lt + h : 0] : ia + h;
        const float4 ta = rel[SOME || active ? ia : tb], tbv = rel[SOME || vb ? ib : tb];
        if (tid == 0) atomicAdd(&counts[1], (unsigned long long)total * (unsigned long long)nt);
        const float2 AX = make_float2(ta.x, ta.x), AY = make_float2(ta.y, ta.y), AZ = make_float2(ta.z, ta.z);
        const float2 BX = make_float2(tbv.x, tbv.x), BY = make_float2(tbv.y, tbv.y), BZ = make_float2(tbv.z, tbv.z);
        float sax = 0.f, say = 0.f, saz = 0.f, eax = 0.f, eay = 0.f, eaz = 0.f;
        float sbx = 0.f, sby = 0.f, sbz = 0.f, ebx = 0.f, eby = 0.f, ebz = 0.f;
        // Sources are staged one tile ahead: the thread's two sources of the
        // next tile are copied into raw[buf] (cp.async) while the current
        // tile's pairs run.  kb / kbeg: the thread's current source box and its
        // first running index; kn: the box slots of the copied sources, -1 past
        // the end.
        int kb = 0, kbeg = 0, kn0 = -1, kn1 = -1;
        auto copy_one = [&](int j, int end, float4 *dst) {
            if (j >= end) return -1;
            int2 rg = sh.nb_rng[kb];
            while (rg.y <= j) {
                kbeg = rg.y;
                rg = sh.nb_rng[++kb];
            }
            cp_async16(dst, rel + rg.x + (j - kbeg));
            return kb;
        };
        auto prefetch = [&](int c0, int buf) {
            const int c1 = min(total, c0 + tile);
            kn0 = copy_one(c0 + tid, c1, &sh.raw[buf][tid]);
            kn1 = copy_one(c0 + kP2PThreads + tid, c1, &sh.raw[buf][kP2PThreads + tid]);
            cp_async_commit();
        };
        // the copied tile, moved to its target-box offset, into the staging rows
        auto stage_one = [&](int kn, int k, int buf) {
            float4 v = pad;
            if (kn >= 0) {
                const float4 r = sh.raw[buf][k];
                const float4 o = sh.nb_off[kn];
                v = make_float4(r.x + o.x, r.y + o.y, r.z + o.z, r.w);
            }
            sh.st[buf][0][k] = -v.x;
            sh.st[buf][1][k] = -v.y;
            sh.st[buf][2][k] = -v.z;
            if (!UQ) sh.st[buf][3][k] = v.w;
        };
        prefetch(0, 0);
        float2 gax = make_float2(0.f, 0.f), gay = gax, gaz = gax, gbx = gax, gby = gax, gbz = gax;
        for (int c0 = 0, buf = 0; c0 < total; c0 += tile, buf ^= 1) {
            cp_async_wait_all();
            stage_one(kn0, tid, buf);
            if (tile > kP2PThreads) stage_one(kn1, kP2PThreads + tid, buf);
            // one barrier per tile: a thread writes st[buf] again two tiles later, after
            // the barrier of the tile between, which every reader of st[buf] reached
            __syncthreads();
            if (c0 + tile < total) prefetch(c0 + tile, buf ^ 1);
            if (active) {
                const float *sx = &sh.st[buf][0][grp * run];
                const float *se = sx + run;
#pragma unroll 1
                for (; sx < se; sx += 8) {
#pragma unroll
                    for (int k = 0; k < 8; k += 2) {
                        const float2 X = ld2(sx, k), Y = ld2(sx + kSrcTile, k), Z = ld2(sx + 2 * kSrcTile, k);
                        const float2 Q = UQ ? make_float2(1.f, 1.f) : ld2(sx + 3 * kSrcTile, k);
                        pair2<CLAMP, UQ>(X, Y, Z, Q, AX, AY, AZ, E2, gax, gay, gaz);
                        pair2<CLAMP, UQ>(X, Y, Z, Q, BX, BY, BZ, E2, gbx, gby, gbz);
                    }
                }
                // 32 sources' FP32 sums per compensated addition (two tiles of a shorter run); 64
                // take 0.4 to 1.3 % less of a step and lose twice as much to each uncompensated sum
                if (run == 32 || buf || c0 + tile >= total) {
                    kahan_add(sax, eax, gax.x + gax.y);
                    kahan_add(say, eay, gay.x + gay.y);
                    kahan_add(saz, eaz, gaz.x + gaz.y);
                    kahan_add(sbx, ebx, gbx.x + gbx.y);
                    kahan_add(sby, eby, gby.x + gby.y);
                    kahan_add(sbz, ebz, gbz.x + gbz.y);
                    gax = gay = gaz = gbx = gby = gbz = make_float2(0.f, 0.f);
                }
            }
        }
        // the groups' sums, through shared memory (the staging rows are free
        // after the barrier): six rows of kP2PThreads
        float(*red)[kP2PThreads] = reinterpret_cast<float(*)[kP2PThreads]>(&sh.st[0][0][0]);
        __syncthreads();
        if (grp > 0 && active) {
            red[0][tid] = sax - eax;
            red[1][tid] = say - eay;
            red[2][tid] = saz - eaz;
            red[3][tid] = sbx - ebx;
            red[4][tid] = sby - eby;
            red[5][tid] = sbz - ebz;
        }
        __syncthreads();
        if (grp == 0) {
            for (int g = 1; g < s; g++) {
                const int t = g * h + lt;
                kahan_add(sax, eax, red[0][t]);
                kahan_add(say, eay, red[1][t]);
                kahan_add(saz, eaz, red[2][t]);
                kahan_add(sbx, ebx, red[3][t]);
                kahan_add(sby, eby, red[4][t]);
                kahan_add(sbz, ebz, red[5][t]);
            }
            const double ca = UQ ? qm[ia] * (double)ta.w : qm[ia];
            ax[ia] = (double)(sax - eax) * ca;
            ay[ia] = (double)(say - eay) * ca;
            az[ia] = (double)(saz - eaz) * ca;
            if (vb) {
                const double c = UQ ? qm[ib] * (double)tbv.w : qm[ib];
                ax[ib] = (double)(sbx - ebx) * c;
                ay[ib] = (double)(sby - eby) * c;
                az[ib] = (double)(sbz - ebz) * c;
            }
        }
        __syncthreads();  // the staging rows and lists are reused
    }
}

// The forest's work items (box, chunk of its targets), largest first by class:
// a plume's densest boxes hold twenty times the mean, and one of their chunks
// started last keeps a few CTAs running after all others (24 plumes 6.09 -> 5.30 ms
// per two steps, 256 plumes 41.7 -> 39.1 ms a step, against boxes in order).  An item's size is
// estimated by targets x particles of its box, for its near boxes are as dense.
// Targets and items per class are counted in one launch; in the next each CTA
// reserves its places in every class.
constexpr int kItemThreads = 256;
// the most items: a box's targets are cut into ceil(targets / 8) chunks at most (p2p_chunks)
inline size_t near_items_room(int n, int boxes) { return (size_t)n / 8 + (size_t)boxes; }
__device__ __forceinline__ int near_item_class(int nt, int np, int chunks) {
    return 31 - __clz((int)min(1ll + (long long)((nt + chunks - 1) / chunks) * np, 0x7fffffffll));
}
__global__ void __launch_bounds__(kWarps * 32)
leaf_targets_kernel(int nbox, const int *__restrict__ nbd, const int *__restrict__ start,
                    const double *__restrict__ qm, int *__restrict__ ntgt, int *__restrict__ classes) {
    __shared__ int cnt[kItemClasses];
    if (threadIdx.x < kItemClasses) cnt[threadIdx.x] = 0;
    __syncthreads();
    SV_WARP_BOXES(kWarps) {
        const int s0 = start[b], s1 = start[b + 1];
        int f = 0;
        for (int j = s0 + lane; j < s1; j += 32) f += qm[j] != 0.0;
        f = __reduce_add_sync(0xffffffffu, f);
        const int c = p2p_chunks(f, 1);
        if (lane == 0) {
            ntgt[b] = f;
            if (c) atomicAdd(&cnt[near_item_class(f, s1 - s0, c)], c);
        }
    }
    __syncthreads();
    if (threadIdx.x < kItemClasses && cnt[threadIdx.x]) atomicAdd(&classes[threadIdx.x], cnt[threadIdx.x]);
}
__global__ void __launch_bounds__(kItemThreads)
near_items_kernel(int nbox, const int *__restrict__ nbd, const int *__restrict__ start,
                  const int *__restrict__ ntgt, const int *__restrict__ classes, int *__restrict__ placed,
                  int *__restrict__ total, int2 *__restrict__ items, int room) {
    __shared__ int cnt[kItemClasses], at[kItemClasses];
    const int tid = threadIdx.x;
    if (tid < kItemClasses) cnt[tid] = 0;
    __syncthreads();
    const int nb = level_boxes(nbox, nbd);
    const int b = blockIdx.x * kItemThreads + tid;  // one box per thread
    const int nt = b < nb ? ntgt[b] : 0, c = p2p_chunks(nt, 1);
    int cls = 0, mine = 0;
    if (c) {
        cls = near_item_class(nt, start[b + 1] - start[b], c);
        mine = atomicAdd(&cnt[cls], c);
    }
    __syncthreads();
    if (tid < kItemClasses) {
        // classes in falling order: those above this one come first
        int before = 0, all = 0;
        for (int k = 0; k < kItemClasses; k++) {
            const int n = classes[k];
            all += n;
            if (k > tid) before += n;
        }
        at[tid] = before + (cnt[tid] ? atomicAdd(&placed[tid], cnt[tid]) : 0);
        if (blockIdx.x == 0 && tid == 0) *total = min(all, room);
    }
    __syncthreads();
    for (int k = 0; k < c; k++) {
        const int o = at[cls] + mine + k;
        if (o < room) items[o] = make_int2(b, k);
    }
}

// A single tree launches one CTA per item (box, part): part p of `parts` takes the
// box's target chunks p, p + parts, ...  LIST: trees with image copies, and the
// forest (list set), one CTA per item (box, chunk) of the list and as many as the
// boxes have room, items past that shared out: a CTA that ends after its item lets
// the far field's kernels in between.  (As many as fit at once, pulling items from a
// queue, held every SM until the list was done and ran the two in turn on small
// batches: 0.71 to 1.0 ms against 0.64 to 0.66 for three balls of 9,000 to 20,000
// ions; 24 and 256 plumes the same within 1 %.)
// Image copies are sources only: a box's targets are gathered first, so that the
// lanes hold no image (three of four particles of a plume on the rotation axis: 24
// plumes, every other one rotational, 5.19 -> 3.2 ms a step).  Without images
// nearly every particle is a target and the kernel is 2 % faster without the
// second form (one million ions, 7.63 against 7.83 ms).
// counts[2] != 0: box_relative_kernel met two different charges.
template <int WS, bool CLAMP, bool LIST>
__global__ void __launch_bounds__(kP2PThreads, 6)
p2p_kernel(int nbox, int parts, const int2 *__restrict__ list, const int *__restrict__ bpid,
           const int *__restrict__ start, const int4 *__restrict__ coord, const int *__restrict__ nbr,
           const double *__restrict__ qm, const double *__restrict__ roots, int level, float eps2,
           double *__restrict__ ax, double *__restrict__ ay, double *__restrict__ az,
           unsigned long long *__restrict__ counts, const int *__restrict__ has_tgt, const float4 *__restrict__ rel,
           const int *__restrict__ fd, const int *__restrict__ fd_cnt, int fd_cap) {
    __shared__ __align__(16) P2PShared<WS> sh;
    const int items = LIST && list ? (int)counts[3] : nbox * parts;
    const int stride = LIST && list ? 1 << 20 : parts;
    const bool uq = counts[2] == 0;
    for (int it = blockIdx.x; it < items; it += gridDim.x) {
        int b = it / parts, part = it - b * parts;
        if (LIST && list) {
            b = list[it].x;
            part = list[it].y;
        }
        const int ntgt = has_tgt[b];
        if (ntgt) {
#define SV_ITEM(U, S) p2p_item<WS, CLAMP, U, S>(sh, b, ntgt, part, parts, stride, bpid, start, coord, nbr, qm, roots, \
                                                level, eps2, ax, ay, az, counts, rel, fd, fd_cnt, fd_cap)
            if (LIST && ntgt < start[b + 1] - start[b]) {
                if (uq) SV_ITEM(true, true);
                else SV_ITEM(false, true);
            } else {
                if (uq) SV_ITEM(true, false);
                else SV_ITEM(false, false);
            }
#undef SV_ITEM
        }
        if (!LIST) return;
        __syncthreads();
    }
}

// P2P launch: well-separation, whether r^2 needs the kMinR2 floor, and whether the tree holds images or comes
// with a list of items
inline void launch_p2p(int ws, bool images, float eps2, int grid, cudaStream_t st, int nbox, int parts,
                       const int2 *list, const int *bpid, const int *start, const int4 *coord, const int *nbr,
                       const double *qm, const double *roots, int level, double *ax, double *ay, double *az,
                       unsigned long long *counts, const int *has_tgt, const float4 *rel, const int *fd = nullptr,
                       const int *fd_cnt = nullptr, int fd_cap = 0) {
    const bool clamp = !(eps2 >= kMinR2), gather = images || list;
#define SV_P2P(W, C, G) p2p_kernel<W, C, G><<<grid, kP2PThreads, 0, st>>>(nbox, parts, list, bpid, start, coord, nbr,  \
                                                                      qm, roots, level, eps2, ax, ay, az, counts, \
                                                                      has_tgt, rel, fd, fd_cnt, fd_cap)
    if (ws == 1) {
        if (clamp) gather ? SV_P2P(1, true, true) : SV_P2P(1, true, false);
        else gather ? SV_P2P(1, false, true) : SV_P2P(1, false, false);
    } else {
        if (clamp) gather ? SV_P2P(2, true, true) : SV_P2P(2, true, false);
        else gather ? SV_P2P(2, false, true) : SV_P2P(2, false, false);
    }
#undef SV_P2P
}

template <int P>
sv_status run_fmm(sv_ctx *c, Fmm &F, Tree &T) {
    constexpr int NC = ncoef(P);
    const int L = T.deepest;
    const int ws = F.ws;
    const int ns1 = 2 * ws + 1, ns = ns1 * ns1 * ns1;
    const int cap = ns * 8 - ns;
    Sorted &S = c->S;
    // arena: per level M, Loc, nbr, m2l, cnt, and M2L partials where a box's list is split
    auto rounded = [](size_t sz) { return (sz + 255) & ~(size_t)255; };
    int chunks[kMortonBits + 1];
    size_t bytes = 0;
    for (int l = 0; l <= L; l++) {
        const size_t nb = T.lv[l].nbox;
        chunks[l] = m2l_chunks((int)nb);
        bytes += 2 * rounded(nb * NC * sizeof(float2)) + rounded(nb * ns * sizeof(int)) +
                 rounded(nb * cap * sizeof(int2)) + rounded(nb * sizeof(int));
        if (chunks[l] > 1) bytes += rounded(nb * chunks[l] * NC * sizeof(float2));
    }
    for (int l = 0; l <= L; l++) bytes += rounded((size_t)T.lv[l].nbox * sizeof(uint64_t));  // box codes
    // far-direct lists of the leaf boxes (sv_params.fmm_direct_pairs; 0: 1024 pairs, < 0: none)
    const int fd_thresh = c->P.fmm_direct_pairs == 0 ? 1024 : c->P.fmm_direct_pairs;
    const bool use_fd = fd_thresh > 0 && L >= 2;
    if (use_fd) bytes += rounded((size_t)T.lv[L].nbox * (kFarDirectCap + 1) * sizeof(int));
    if (F.arena_bytes < bytes) {
        cudaFree(F.arena);
        F.arena = nullptr;
        F.arena_bytes = 0;
        const size_t want = bytes + bytes / 2;  // headroom: a growing tree reallocates rarely
        SV_CK(c, cudaMalloc(&F.arena, want));
        F.arena_bytes = want;
    }
    char *p = (char *)F.arena;
    auto carve = [&](size_t sz) {
        char *r = p;
        p += (sz + 255) & ~(size_t)255;
        return (void *)r;
    };
    float2 *Mv[kMortonBits + 1], *Lv[kMortonBits + 1], *part[kMortonBits + 1];
    int *nbr[kMortonBits + 1], *cnt[kMortonBits + 1];
    int2 *lst[kMortonBits + 1];
    for (int l = 0; l <= L; l++) {
        const size_t nb = T.lv[l].nbox;
        Mv[l] = (float2 *)carve(nb * NC * sizeof(float2));
        Lv[l] = (float2 *)carve(nb * NC * sizeof(float2));
        nbr[l] = (int *)carve(nb * ns * sizeof(int));
        lst[l] = (int2 *)carve(nb * cap * sizeof(int2));
        cnt[l] = (int *)carve(nb * sizeof(int));
        part[l] = chunks[l] > 1 ? (float2 *)carve(nb * chunks[l] * NC * sizeof(float2)) : Lv[l];
    }
    // which boxes hold targets (all of them unless symmetry images are present)
    int *tgt[kMortonBits + 1];
    {
        int64_t tot = 0;
        for (int l = 0; l <= L; l++) tot += T.lv[l].nbox;
        if (F.tgt_cap < tot) {
            cudaFree(F.has_tgt);
            F.has_tgt = nullptr;
            const int64_t want = tot + tot / 2;  // headroom: a growing tree reallocates rarely
            SV_CK(c, cudaMalloc(&F.has_tgt, sizeof(int) * want));
            F.tgt_cap = want;
        }
        int64_t o = 0;
        for (int l = 0; l <= L; l++) {
            tgt[l] = F.has_tgt + o;
            o += T.lv[l].nbox;
        }
    }
    // every level's lists in two launches (near lists, then interaction lists)
    ListArgs la{};
    la.nlev = L + 1;
    for (int l = 0; l <= L; l++) {
        ListLevel &q = la.lv[l];
        q.nbox = T.lv[l].nbox;
        q.first = la.total;
        la.total += q.nbox;
        q.coord = T.lv[l].coord;
        q.code = (uint64_t *)carve((size_t)q.nbox * sizeof(uint64_t));
        q.nbr = nbr[l];
        q.parent = T.lv[l].parent;
        q.pchild0 = l > 0 ? T.lv[l - 1].child0 : nullptr;
        q.pnbr = l > 0 ? nbr[l - 1] : nullptr;
        q.m2l = lst[l];
        q.m2l_cnt = cnt[l];
        q.start = T.lv[l].start;
        q.fd = q.fd_cnt = nullptr;
    }
    la.fd_cap = kFarDirectCap;
    la.fd_thresh = fd_thresh;
    la.trim = F.trim;
    if (use_fd) {
        la.lv[L].fd = (int *)carve((size_t)T.lv[L].nbox * kFarDirectCap * sizeof(int));
        la.lv[L].fd_cnt = (int *)carve((size_t)T.lv[L].nbox * sizeof(int));
    }
    phase_mark(c, 2);
    SV_CK(c, cudaMemsetAsync(F.d_counts, 0, kCounts * sizeof(unsigned long long), c->stream));
    if (F.rel_cap < c->S.n) {
        cudaFree(F.rel);
        cudaFree(F.far);
        F.rel = nullptr;
        F.far = nullptr;
        SV_CK(c, cudaMalloc(&F.rel, sizeof(float4) * c->S.n));
        SV_CK(c, cudaMalloc(&F.far, 3 * sizeof(double) * c->S.n));
        F.rel_cap = c->S.n;
    }
    double *fx = F.far, *fy = F.far + F.rel_cap, *fz = F.far + 2 * F.rel_cap;
    // Two streams from here on.  The second takes the near and interaction
    // lists of every level in two
    // launches (boxes found by binary search over each level's Morton codes),
    // then runs the near field (P2P), which needs only the sorted particles,
    // the leaf boxes, their target flags and near lists, and writes the
    // accelerations.  The main stream runs the
    // upward pass, then M2L / L2L and the far field (L2P or the treecode's M2P, into their
    // own arrays) beside the near field, then waits for it; the scatter to the
    // caller's order adds the two.
    SV_CK(c, cudaEventRecord(F.ev_fork, c->stream));
    SV_CK(c, cudaStreamWaitEvent(F.side, F.ev_fork, 0));
    {
        const Level &V = T.lv[L];
        box_codes_kernel<<<div_up(la.total, 256), 256, 0, F.side>>>(la);
        SV_LAUNCHED(c);
        const int64_t slots = (int64_t)la.total * ns;
        if (ws == 1) near_lists_kernel<1><<<div_up(slots, 256), 256, 0, F.side>>>(la);
        else near_lists_kernel<2><<<div_up(slots, 256), 256, 0, F.side>>>(la);
        SV_LAUNCHED(c);
        if (L > 0) {
            const int g = std::min(div_up(la.total - la.lv[1].first, kWarps), 16 * device_sms());
            if (ws == 1) m2l_lists_kernel<1><<<g, kWarps * 32, 0, F.side>>>(la, cap, F.d_counts);
            else m2l_lists_kernel<2><<<g, kWarps * 32, 0, F.side>>>(la, cap, F.d_counts);
            SV_LAUNCHED(c);
        }
        SV_CK(c, cudaEventRecord(F.ev_lists, F.side));
        box_relative_kernel<<<div_up(V.nbox, kWarps), kWarps * 32, 0, F.side>>>(
            V.nbox, nullptr, nullptr, V.start, V.coord, S.x, S.y, S.z, S.q, S.root, L, F.rel, F.d_counts + 2, S.qm,
            tgt[L]);
        SV_LAUNCHED(c);
        SV_CK(c, cudaEventRecord(F.ev_rel, F.side));
        if (c->P.profile_phases) SV_CK(c, cudaEventRecord(F.ev_near[0], F.side));
        // few boxes: their target chunks to several CTAs, two waves of the CTAs that fit at once
        const int parts = std::max(1, std::min(8, div_up(2 * 6 * device_sms(), V.nbox)));
        launch_p2p(ws, c->P.symmetry != SV_SYM_NONE, (float)c->P.softening2, V.nbox * parts, F.side, V.nbox, parts, nullptr, nullptr, V.start,
                   V.coord, nbr[L], S.qm, S.root, L, S.ax, S.ay, S.az, F.d_counts, tgt[L], F.rel, la.lv[L].fd,
                   la.lv[L].fd_cnt, kFarDirectCap);
        SV_LAUNCHED(c);
        if (c->P.profile_phases) {
            SV_CK(c, cudaEventRecord(F.ev_near[1], F.side));
            c->near_ev[0] = F.ev_near[0];
            c->near_ev[1] = F.ev_near[1];
        }
        SV_CK(c, cudaEventRecord(F.ev_join, F.side));
    }
    phase_mark(c, 3);
    // Upward pass.  Beside the lists it holds SMs that the lists, and behind them the near
    // field, the longest kernel of an evaluation, are waiting for; after them it
    // starts late.  It waits where the near field is long: in trees of four boxes per
    // level or more (balls of 8,000 to a million ions, orders 6 and 8: 0.97 to 1.03 of the
    // time at once, 0.99 on average), and in columns of 64 leaf boxes per SM or more
    // (0.99 to 1.04 at 350,000 and 420,000 ions, 0.97 to 1.00 from 500,000 to a million).
    // Smaller columns start at once: waiting takes 1.03 to 1.10 of the time up to
    // 65,000 ions, 0.99 to 1.05 up to 300,000.
    if (T.lv[L].nbox >= 64 * device_sms() || (int64_t)T.lv[L].nbox >= int64_t(1) << 2 * L)
        SV_CK(c, cudaStreamWaitEvent(c->stream, F.ev_lists, 0));
    {
        const Level &V = T.lv[L];
        p2m_kernel<P><<<div_up(V.nbox, p2m_warps<P>()), p2m_warps<P>() * 32, 0, c->stream>>>(
            V.nbox, nullptr, nullptr, V.start, V.coord, S.x, S.y, S.z, S.q, S.root, L, F.nrm, Mv[L]);
        SV_LAUNCHED(c);
    }
    // levels 2 .. coarse and their children have few boxes: one launch for all of them
    int coarse = 1;
    while (coarse + 1 < L && T.lv[coarse + 2].nbox <= kCoarseBoxes) coarse++;
    if (coarse == 2) coarse = 1;  // one level gains nothing from one CTA
    for (int l = L - 1; l > coarse; l--) {
        const Level &V = T.lv[l];
        m2m_kernel<P><<<div_up(V.nbox, kWarps), kWarps * 32, 0, c->stream>>>(
            V.nbox, nullptr, V.child0, T.lv[l + 1].coord, Mv[l + 1], Mv[l], F.otab);
        SV_LAUNCHED(c);
    }
    if (coarse >= 2) {
        CoarseM2M cm{};
        cm.top = coarse;
        cm.last = 2;
        cm.otab = F.otab;
        for (int l = 2; l <= coarse + 1; l++) {
            cm.nbox[l] = T.lv[l].nbox;
            cm.child0[l] = T.lv[l].child0;
            cm.coord[l] = T.lv[l].coord;
            cm.M[l] = Mv[l];
            cm.tmp[l] = Lv[l];  // free until the downward pass
        }
        SV_CK(c, (dyn_smem<P>(m2m_coarse_kernel<P>)));
        m2m_coarse_kernel<P><<<1, kCoarseWarps * 32, coarse_smem<P>(), c->stream>>>(cm);
        SV_LAUNCHED(c);
    }
    // the second stream's lists, leaf offsets and leaf flags; then the coarser flags
    SV_CK(c, cudaStreamWaitEvent(c->stream, F.ev_rel, 0));
    TargetArgs tf{};
    tf.L = L;
    tf.done = reinterpret_cast<unsigned *>(F.d_counts + 4);
    for (int l = 0; l <= L; l++) {
        tf.nbox[l] = T.lv[l].nbox;
        tf.child0[l] = T.lv[l].child0;
        tf.flag[l] = tgt[l];
        if (l == 0 || (l < L && T.lv[l].nbox <= kFlagTop * device_sms())) tf.top = l;
    }
    target_flags_kernel<<<T.lv[tf.top].nbox, kFlagThreads, 0, c->stream>>>(tf);
    SV_LAUNCHED(c);
    phase_mark(c, 4);
    const bool treecode = c->P.fmm_type == SV_FMM_TREECODE || c->P.fmm_type == SV_FMM_TREECODE_OUTLIERS;
    // downward pass: M2L of all levels in one launch, then L2L level by level
    // (the treecode evaluates multipoles at the particles instead)
    F.tc.launched = false;
    if (!treecode && L >= 2) {
        M2LArgs a{};
        a.cap = cap;
        a.esz = F.H.esz;
        a.osz = F.H.osz;
        a.dsz = F.H.dsz;
        a.eps2 = c->P.softening2;
        a.root = S.root;
        a.cls_theta = F.cls_theta;
        a.cls_phase = F.cls_phase;
        a.cls_rho2 = F.cls_rho2;
        a.dmat = F.dmat;
        a.zc = F.zc;
        int warps = 0;
        for (int l = 2; l <= L; l++) {
            M2LLevel &V = a.lv[a.nlev++];
            V.nbox = T.lv[l].nbox;
            V.chunks = chunks[l];
            V.warp0 = warps;
            V.level = l;
            V.nbd = nullptr;
            V.bpid = nullptr;
            V.m2l = lst[l];
            V.cnt = cnt[l];
            V.has_tgt = tgt[l];
            V.M = Mv[l];
            V.out = part[l];
            warps += V.nbox * V.chunks;
        }
        if (c->P.fmm_m2l_tc >= 0) {
            // the tensor-core M2L; the rotation kernel below runs only if it overflowed its room
            TcArgs ta{};
            ta.nlev = a.nlev;
            ta.cap = cap;
            ta.eps2 = c->P.softening2;
            ta.root = S.root;
            ta.cls_rho2 = F.cls_rho2;
            int64_t boxes = 0;
            for (int k = 0; k < a.nlev; k++) {
                const M2LLevel &V = a.lv[k];
                TcLevel &q = ta.lv[k];
                q.nbox = V.nbox;
                q.level = V.level;
                q.chunks = V.chunks;
                q.warp0 = V.warp0;
                q.first = (int)boxes;
                q.nbd = nullptr;
                q.bpid = nullptr;
                q.m2l = lst[V.level];
                q.cnt = V.cnt;
                q.has_tgt = V.has_tgt;
                q.M = V.M;
                q.out = V.out;
                boxes += V.nbox;
            }
            ta.total_boxes = (int)boxes;
            // room: the last evaluation's translations (read back by then) with a margin, at least 32 per box
            const int64_t last = F.tc.h_ctl && F.tc.p == P && F.tc.ws == ws ? F.tc.h_ctl[0] : 0;
            SV_TRY(m2l_tc_prepare(c, F.tc, P, ws, std::max<int64_t>(last + last / 4, 32 * boxes)));
            ta.ncls = F.tc.ncls;
            SV_TRY(m2l_tc_launch(c, F.tc, ta, warps, c->stream));
            a.run_if = m2l_tc_skip_flag(F.tc);
            F.tc.launched = true;
        }
        m2l_kernel<P><<<div_up(warps, m2l_warps<P>()), m2l_warps<P>() * 32, 0, c->stream>>>(a);
        SV_LAUNCHED(c);
        CoarseL2L cl{};
        // the same for the locals: a warp per box
        int lcoarse = 1;
        while (lcoarse + 1 <= L && T.lv[lcoarse + 1].nbox <= kCoarseBoxes) lcoarse++;
        if (lcoarse == 2) lcoarse = 1;  // one level gains nothing from one CTA
        cl.first = 2;
        cl.last = lcoarse;
        for (int l = 2; l <= L; l++) {
            const Level &V = T.lv[l];
            L2LArgs &b = cl.lv[l];
            b.nbox = V.nbox;
            b.chunks = chunks[l];
            b.has_parent = l > 2;
            b.nbd = nullptr;
            b.parent = V.parent;
            b.coord = V.coord;
            b.has_tgt = tgt[l];
            b.Lp = l > 2 ? Lv[l - 1] : nullptr;
            b.part = part[l];
            b.L = Lv[l];
            b.otab = F.otab;
        }
        if (lcoarse >= 2) {
            SV_CK(c, (dyn_smem<P>(l2l_coarse_kernel<P>)));
            l2l_coarse_kernel<P><<<1, kCoarseWarps * 32, coarse_smem<P>(), c->stream>>>(cl);
            SV_LAUNCHED(c);
        }
        for (int l = std::max(2, lcoarse + 1); l <= L; l++) {
            l2l_kernel<P><<<div_up(T.lv[l].nbox, kWarps), kWarps * 32, 0, c->stream>>>(cl.lv[l]);
            SV_LAUNCHED(c);
        }
    }
    phase_mark(c, 5);
    // far field into its own arrays, beside the near field
    S.far = nullptr;
    {
        const Level &V = T.lv[L];
        if (L >= 2 && treecode) {
            TreecodeArgs ta{};
            ta.L = L;
            ta.cap = cap;
            ta.ws = ws;
            ta.nleaf = V.nbox;
            for (int l = 0; l <= L; l++) {
                ta.parent[l] = T.lv[l].parent;
                ta.coord[l] = T.lv[l].coord;
                ta.m2l[l] = lst[l];
                ta.m2l_cnt[l] = cnt[l];
                ta.M[l] = Mv[l];
            }
            ta.leaf_start = V.start;
            ta.has_tgt = tgt[L];
            ta.x = S.x;
            ta.y = S.y;
            ta.z = S.z;
            ta.qm = S.qm;
            ta.root = S.root;
            ta.nrm = F.nrm;
            ta.eps2 = c->P.softening2;
            ta.ax = fx;
            ta.ay = fy;
            ta.az = fz;
            ta.accumulate = 0;
            m2p_kernel<P><<<div_up(V.nbox, kWarps), kWarps * 32, 0, c->stream>>>(ta);
            SV_LAUNCHED(c);
            S.far = F.far;
        } else if (L >= 2) {
            l2p_kernel<P><<<div_up(V.nbox, kWarps), kWarps * 32, 0, c->stream>>>(
                V.nbox, nullptr, nullptr, V.start, F.rel, S.qm, S.root, L, F.nrm, Lv[L], fx, fy, fz, tgt[L], 0);
            SV_LAUNCHED(c);
            S.far = F.far;
        }
        S.far_stride = F.rel_cap;
        phase_mark(c, 6);
    }
    SV_CK(c, cudaStreamWaitEvent(c->stream, F.ev_join, 0));
    SV_CK(c, cudaMemcpyAsync(F.h_counts, F.d_counts, 2 * sizeof(unsigned long long), cudaMemcpyDeviceToHost,
                             c->stream));
    c->stats.levels = L;
    c->stats.boxes = T.lv[L].nbox;
    return SV_OK;
}


// ------------------------------------------------------------------ forest --

inline int forest_grid(int cap, int per_cta) {
    const int g = div_up(cap > 0 ? cap : 1, per_cta);
    const int gmax = 16 * device_sms();  // grid-stride launches: at most 16 CTAs per SM
    return g < gmax ? g : gmax;
}

template <int P>
sv_status run_fmm_forest(sv_ctx *c, Fmm &F, const ForestArgs &fa) {
    const ForestSpec &f = fa.spec;
    const int L = f.L;
    const int ws = F.ws;
    const int ns1 = 2 * ws + 1, ns = ns1 * ns1 * ns1;
    const int cap = ns * 8 - ns;
    Sorted &S = c->S;
    Tree &T = *F.ftree;
    int *nbd = fa.d_nbox;
    SV_TRY(tree_build_forest(c, T, f, nbd, fa.d_err));
    SV_CK(c, cudaMemsetAsync(F.d_counts, 0, kCounts * sizeof(unsigned long long), c->stream));
    // Two streams, as in run_fmm: target flags, lists and the near field on the
    // second (the forest's slots only: the direct plumes' slots belong to
    // another stream), the upward and downward passes on the main one.
    cudaStream_t sd = F.side;
    SV_CK(c, cudaEventRecord(F.ev_fork, c->stream));
    SV_CK(c, cudaStreamWaitEvent(sd, F.ev_fork, 0));
    root_nbr_kernel<<<forest_grid(f.cap[0] * ns, 256), 256, 0, sd>>>(F.fnbr[0], ns, f.cap[0], nbd);
    SV_LAUNCHED(c);
    int *classes = reinterpret_cast<int *>(F.d_counts + 5);
    leaf_targets_kernel<<<forest_grid(f.cap[L], kWarps), kWarps * 32, 0, sd>>>(f.cap[L], nbd + L, T.lv[L].start, S.qm,
                                                                             F.ftgt[L], classes);
    SV_LAUNCHED(c);
    for (int l = L - 1; l >= 0; l--) {
        parent_targets_kernel<<<forest_grid(f.cap[l], 256), 256, 0, sd>>>(f.cap[l], nbd + l, T.lv[l].child0,
                                                                        F.ftgt[l + 1], F.ftgt[l]);
        SV_LAUNCHED(c);
    }
    // far-direct lists at the leaf level (sv_params.fmm_direct_pairs, as the single tree's)
    const int fd_thresh = c->P.fmm_direct_pairs == 0 ? 1024 : c->P.fmm_direct_pairs;
    for (int l = 1; l <= L; l++) {
        const Level &V = T.lv[l];
        const Level &U = T.lv[l - 1];
        const bool fdl = l == L && fd_thresh > 0;
        if (ws == 1)
            build_lists_kernel<1><<<forest_grid(f.cap[l], kWarps), kWarps * 32, 0, sd>>>(
                f.cap[l], nbd + l, V.parent, V.coord, F.fnbr[l - 1], U.child0, F.fnbr[l], F.flst[l], F.fcnt[l], cap,
                F.trim, F.d_counts, V.start, fdl ? F.ffd : nullptr, F.ffd_cnt, kFarDirectCap, fd_thresh);
        else
            build_lists_kernel<2><<<forest_grid(f.cap[l], kWarps), kWarps * 32, 0, sd>>>(
                f.cap[l], nbd + l, V.parent, V.coord, F.fnbr[l - 1], U.child0, F.fnbr[l], F.flst[l], F.fcnt[l], cap,
                F.trim, F.d_counts, V.start, fdl ? F.ffd : nullptr, F.ffd_cnt, kFarDirectCap, fd_thresh);
        SV_LAUNCHED(c);
    }
    SV_CK(c, cudaEventRecord(F.ev_lists, sd));
    {
        const Level &V = T.lv[L];
        const int g = forest_grid(f.cap[L], kWarps);
        SV_CK(c, cudaMemsetAsync(S.ax, 0, sizeof(double) * f.n, sd));
        SV_CK(c, cudaMemsetAsync(S.ay, 0, sizeof(double) * f.n, sd));
        SV_CK(c, cudaMemsetAsync(S.az, 0, sizeof(double) * f.n, sd));
        box_relative_kernel<<<g, kWarps * 32, 0, sd>>>(f.cap[L], nbd + L, V.pid, V.start, V.coord, S.x, S.y, S.z,
                                                       S.q, fa.roots, L, F.frel, F.d_counts + 2);
        SV_LAUNCHED(c);
        near_items_kernel<<<std::max(1, div_up(f.cap[L], kItemThreads)), kItemThreads, 0, sd>>>(
            f.cap[L], nbd + L, V.start, F.ftgt[L], classes, classes + kItemClasses,
            reinterpret_cast<int *>(F.d_counts + 3), F.fitems, (int)near_items_room(f.n, f.cap[L]));
        SV_LAUNCHED(c);
        launch_p2p(ws, true, (float)c->P.softening2, f.cap[L], sd, f.cap[L], 1, F.fitems, V.pid,
                   V.start, V.coord, F.fnbr[L], S.qm, fa.roots, L, S.ax, S.ay, S.az, F.d_counts, F.ftgt[L], F.frel,
                   fd_thresh > 0 ? F.ffd : nullptr, F.ffd_cnt, kFarDirectCap);
        SV_LAUNCHED(c);
        SV_CK(c, cudaEventRecord(F.ev_join, sd));
    }
    {
        const Level &V = T.lv[L];
        p2m_kernel<P><<<forest_grid(f.cap[L], p2m_warps<P>()), p2m_warps<P>() * 32, 0, c->stream>>>(
            f.cap[L], nbd + L, V.pid, V.start, V.coord, S.x, S.y, S.z, S.q, fa.roots, L, F.nrm, F.fM[L]);
        SV_LAUNCHED(c);
    }
    for (int l = L - 1; l >= 2; l--) {
        const Level &V = T.lv[l];
        m2m_kernel<P><<<forest_grid(f.cap[l], kWarps), kWarps * 32, 0, c->stream>>>(
            f.cap[l], nbd + l, V.child0, T.lv[l + 1].coord, F.fM[l + 1], F.fM[l], F.otab);
        SV_LAUNCHED(c);
    }
    SV_CK(c, cudaStreamWaitEvent(c->stream, F.ev_lists, 0));
    {
        M2LArgs a{};
        a.cap = cap;
        a.esz = F.H.esz;
        a.osz = F.H.osz;
        a.dsz = F.H.dsz;
        a.eps2 = c->P.softening2;
        a.root = fa.roots;
        a.cls_theta = F.cls_theta;
        a.cls_phase = F.cls_phase;
        a.cls_rho2 = F.cls_rho2;
        a.dmat = F.dmat;
        a.zc = F.zc;
        long long warps = 0;
        for (int l = 2; l <= L; l++) {
            M2LLevel &V = a.lv[a.nlev++];
            V.nbox = f.cap[l];
            V.chunks = F.fchunks[l];
            V.warp0 = (int)warps;
            V.level = l;
            V.nbd = nbd + l;
            V.bpid = T.lv[l].pid;
            V.m2l = F.flst[l];
            V.cnt = F.fcnt[l];
            V.has_tgt = F.ftgt[l];
            V.M = F.fM[l];
            V.out = F.fpart[l];
            warps += (long long)V.nbox * V.chunks;
        }
        F.tc.launched = false;
        if (c->P.fmm_m2l_tc >= 0 && F.tc.cap > 0 && F.tc.p == P && F.tc.ws == ws) {
            // the tensor-core M2L (room reserved with the forest); the rotation
            // kernel below runs only if the translations overflowed it
            TcArgs ta{};
            ta.nlev = a.nlev;
            ta.cap = cap;
            ta.eps2 = c->P.softening2;
            ta.root = fa.roots;
            ta.cls_rho2 = F.cls_rho2;
            ta.ncls = F.tc.ncls;
            long long boxes = 0;
            for (int k = 0; k < a.nlev; k++) {
                const M2LLevel &V = a.lv[k];
                TcLevel &q = ta.lv[k];
                q.nbox = V.nbox;
                q.level = V.level;
                q.chunks = V.chunks;
                q.warp0 = V.warp0;
                q.first = (int)boxes;
                q.nbd = V.nbd;
                q.bpid = V.bpid;
                q.m2l = F.flst[V.level];
                q.cnt = V.cnt;
                q.has_tgt = V.has_tgt;
                q.M = V.M;
                q.out = V.out;
                boxes += V.nbox;
            }
            ta.total_boxes = (int)boxes;
            SV_TRY(m2l_tc_launch(c, F.tc, ta, (int)warps, c->stream));
            a.run_if = m2l_tc_skip_flag(F.tc);
            F.tc.launched = true;
        }
        m2l_kernel<P><<<(int)((warps + m2l_warps<P>() - 1) / m2l_warps<P>()), m2l_warps<P>() * 32, 0,
                          c->stream>>>(a);
        SV_LAUNCHED(c);
        for (int l = 2; l <= L; l++) {
            const Level &V = T.lv[l];
            L2LArgs b{};
            b.nbox = f.cap[l];
            b.chunks = F.fchunks[l];
            b.has_parent = l > 2;
            b.nbd = nbd + l;
            b.parent = V.parent;
            b.coord = V.coord;
            b.has_tgt = F.ftgt[l];
            b.Lp = l > 2 ? F.fL[l - 1] : nullptr;
            b.part = F.fpart[l];
            b.L = F.fL[l];
            b.otab = F.otab;
            l2l_kernel<P><<<forest_grid(f.cap[l], kWarps), kWarps * 32, 0, c->stream>>>(b);
            SV_LAUNCHED(c);
        }
    }
    SV_CK(c, cudaStreamWaitEvent(c->stream, F.ev_join, 0));
    {
        const Level &V = T.lv[L];
        const int g = forest_grid(f.cap[L], kWarps);
        l2p_kernel<P><<<g, kWarps * 32, 0, c->stream>>>(f.cap[L], nbd + L, V.pid, V.start, F.frel, S.qm, fa.roots,
                                                        L, F.nrm, F.fL[L], S.ax, S.ay, S.az, F.ftgt[L], 1);
        SV_LAUNCHED(c);
    }
    SV_CK(c, cudaMemcpyAsync(F.h_counts, F.d_counts, 2 * sizeof(unsigned long long), cudaMemcpyDeviceToHost,
                             c->stream));
    return SV_OK;
}

sv_status ensure_tables(sv_ctx *c, Fmm &F, int p, int ws) {
    if (F.p == p && F.ws == ws && F.dmat) return SV_OK;
    std::string err;
    if (!build_fmm_tables(p, ws, F.H, err)) return set_error(c, SV_ERR_INVALID, "FMM tables: %s", err.c_str());
    cudaFree(F.cls_theta); cudaFree(F.cls_phase); cudaFree(F.cls_rho2); cudaFree(F.dmat);
    cudaFree(F.zc); cudaFree(F.nrm); cudaFree(F.otab);
    const FmmTables &H = F.H;
    SV_CK(c, cudaMalloc(&F.cls_theta, sizeof(int) * H.cls_theta.size()));
    SV_CK(c, cudaMalloc(&F.cls_phase, sizeof(float) * H.cls_phase.size()));
    SV_CK(c, cudaMalloc(&F.cls_rho2, sizeof(float) * H.cls_rho2.size()));
    SV_CK(c, cudaMalloc(&F.dmat, sizeof(float) * H.dmat.size()));
    SV_CK(c, cudaMalloc(&F.zc, sizeof(float) * H.zc.size()));
    SV_CK(c, cudaMalloc(&F.nrm, sizeof(float) * H.nrm.size()));
    SV_CK(c, cudaMalloc(&F.otab, sizeof(float) * H.otab.size()));
    SV_CK(c, cudaMemcpy(F.cls_theta, H.cls_theta.data(), sizeof(int) * H.cls_theta.size(), cudaMemcpyHostToDevice));
    SV_CK(c, cudaMemcpy(F.cls_phase, H.cls_phase.data(), sizeof(float) * H.cls_phase.size(), cudaMemcpyHostToDevice));
    SV_CK(c, cudaMemcpy(F.cls_rho2, H.cls_rho2.data(), sizeof(float) * H.cls_rho2.size(), cudaMemcpyHostToDevice));
    SV_CK(c, cudaMemcpy(F.dmat, H.dmat.data(), sizeof(float) * H.dmat.size(), cudaMemcpyHostToDevice));
    SV_CK(c, cudaMemcpy(F.zc, H.zc.data(), sizeof(float) * H.zc.size(), cudaMemcpyHostToDevice));
    SV_CK(c, cudaMemcpy(F.nrm, H.nrm.data(), sizeof(float) * H.nrm.size(), cudaMemcpyHostToDevice));
    SV_CK(c, cudaMemcpy(F.otab, H.otab.data(), sizeof(float) * H.otab.size(), cudaMemcpyHostToDevice));
    F.p = p;
    F.ws = ws;
    return SV_OK;
}

}  // namespace

void fmm_free(sv_ctx *c) {
    if (!c->fmm) return;
    Fmm &F = *c->fmm;
    cudaFree(F.cls_theta); cudaFree(F.cls_phase); cudaFree(F.cls_rho2); cudaFree(F.dmat);
    cudaFree(F.zc); cudaFree(F.nrm); cudaFree(F.otab); cudaFree(F.arena); cudaFree(F.d_counts);
    cudaFree(F.ex); cudaFree(F.ey); cudaFree(F.ez); cudaFree(F.eq); cudaFree(F.em); cudaFree(F.est);
    cudaFree(F.has_tgt); cudaFree(F.rel); cudaFree(F.far);
    cudaFree(F.farena); cudaFree(F.frel);
    m2l_tc_free(F.tc);
    if (F.ftree) {
        tree_release(*F.ftree);
        delete F.ftree;
    }
    cudaFreeHost(F.h_counts);
    if (F.side) cudaStreamDestroy(F.side);
    if (F.ev_fork) cudaEventDestroy(F.ev_fork);
    if (F.ev_join) cudaEventDestroy(F.ev_join);
    if (F.ev_lists) cudaEventDestroy(F.ev_lists);
    if (F.ev_rel) cudaEventDestroy(F.ev_rel);
    for (cudaEvent_t e : F.ev_near)
        if (e) cudaEventDestroy(e);
    c->near_ev[0] = c->near_ev[1] = nullptr;
    delete c->fmm;
    c->fmm = nullptr;
}

static sv_status fmm_state(sv_ctx *c) {
    if (!c->fmm) {
        c->fmm = new Fmm();
        Fmm &F = *c->fmm;
        SV_CK(c, cudaMalloc(&F.d_counts, kCounts * sizeof(unsigned long long)));
        SV_CK(c, cudaMallocHost(&F.h_counts, 2 * sizeof(unsigned long long)));
        SV_CK(c, cudaStreamCreateWithFlags(&F.side, cudaStreamNonBlocking));
        SV_CK(c, cudaEventCreateWithFlags(&F.ev_fork, cudaEventDisableTiming));
        SV_CK(c, cudaEventCreateWithFlags(&F.ev_join, cudaEventDisableTiming));
        SV_CK(c, cudaEventCreateWithFlags(&F.ev_lists, cudaEventDisableTiming));
        SV_CK(c, cudaEventCreateWithFlags(&F.ev_rel, cudaEventDisableTiming));
        SV_CK(c, cudaEventCreate(&F.ev_near[0]));
        SV_CK(c, cudaEventCreate(&F.ev_near[1]));
    }
    return SV_OK;
}

sv_status fmm_sort_images(sv_ctx *c, int64_t first, int64_t last) {
    SV_TRY(fmm_state(c));
    Fmm &F = *c->fmm;
    const int64_t n = c->n;
    int kind = 0, nimg = 1;
    const double *off = nullptr;
    if (c->P.symmetry == SV_SYM_ROTATIONAL) {
        kind = 1;
        nimg = 4;
    } else if (c->P.symmetry == SV_SYM_TRANSLATIONAL) {
        const ImageSet *I = nullptr;
        SV_TRY(image_set(c, &I));
        kind = 2;
        nimg = I->count;
        off = I->zero_first;
    }
    const int64_t ne = n * nimg;
    if (ne > (int64_t)INT32_MAX) return set_error(c, SV_ERR_CAPACITY, "%lld particles with images", (long long)ne);
    if (F.ecap < ne) {
        cudaFree(F.ex); cudaFree(F.ey); cudaFree(F.ez); cudaFree(F.eq); cudaFree(F.em); cudaFree(F.est);
        F.ex = F.ey = F.ez = F.eq = F.em = nullptr;
        F.est = nullptr;
        SV_CK(c, cudaMalloc(&F.ex, sizeof(double) * ne));
        SV_CK(c, cudaMalloc(&F.ey, sizeof(double) * ne));
        SV_CK(c, cudaMalloc(&F.ez, sizeof(double) * ne));
        SV_CK(c, cudaMalloc(&F.eq, sizeof(double) * ne));
        SV_CK(c, cudaMalloc(&F.em, sizeof(double) * ne));
        SV_CK(c, cudaMalloc(&F.est, sizeof(int32_t) * ne));
        F.ecap = ne;
    }
    expand_images_kernel<<<div_up(ne, 256), 256, 0, c->stream>>>(c->x, c->y, c->z, c->q, c->m, force_status(c), n, kind,
                                                                 nimg, off, F.ex, F.ey, F.ez, F.eq, F.em, F.est);
    SV_LAUNCHED(c);
    const ParticleView v{F.ex, F.ey, F.ez, F.eq, F.em, F.est, ne, n};
    return sort_view(c, v, first, last);
}

int fmm_sort_levels(const sv_ctx *c) {
    const int h = c->fmm ? c->fmm->level_hint : -1;
    return h >= 2 ? std::min(kMortonBits, h + 1) : kMortonBits;
}

sv_status fmm_accel(sv_ctx *c) {
    if (c->P.precision != SV_PREC_MIXED)
        return set_error(c, SV_ERR_UNSUPPORTED, "FMM runs in mixed precision only");
    const int p = c->P.fmm_order;
    if (p != 4 && p != 6 && p != 8 && p != 10)
        return set_error(c, SV_ERR_UNSUPPORTED, "FMM order %d not instantiated (4, 6, 8, 10)", p);
    SV_TRY(fmm_state(c));
    Fmm &F = *c->fmm;
    SV_TRY(ensure_tables(c, F, p, c->P.fmm_ws));
    F.trim = c->P.fmm_near == 2 && c->P.fmm_ws == 2;
    Tree *T = nullptr;
    c->S.resort = false;
    SV_TRY(tree_build(c, kDepthMeanOccupancy, c->P.fmm_leaf_target, &T));
    // the depth rule's box counts are exact down to the sorted levels only; a
    // leaf level at or below them needs the full order
    if (T->n_act > 0 && T->deepest >= c->S.key_levels && c->S.key_levels < kMortonBits) {
        c->S.resort = true;
        return SV_OK;
    }
    F.level_hint = T->deepest;
    if (T->n_act == 0) {
        SV_CK(c, cudaMemsetAsync(c->S.ax, 0, sizeof(double) * c->S.n, c->stream));
        SV_CK(c, cudaMemsetAsync(c->S.ay, 0, sizeof(double) * c->S.n, c->stream));
        SV_CK(c, cudaMemsetAsync(c->S.az, 0, sizeof(double) * c->S.n, c->stream));
        return SV_OK;
    }
    switch (p) {
    case 4: SV_TRY(run_fmm<4>(c, F, *T)); break;
    case 6: SV_TRY(run_fmm<6>(c, F, *T)); break;
    case 8: SV_TRY(run_fmm<8>(c, F, *T)); break;
    default: SV_TRY(run_fmm<10>(c, F, *T)); break;
    }
    return SV_OK;
}

sv_status fmm_forest_reserve(sv_ctx *c, const ForestArgs &fa) {
    const int p = fa.p;
    if (p != 4 && p != 6 && p != 8 && p != 10)
        return set_error(c, SV_ERR_UNSUPPORTED, "FMM order %d not instantiated (4, 6, 8, 10)", p);
    if (fa.ws != 1 && fa.ws != 2) return set_error(c, SV_ERR_INVALID, "well-separation must be 1 or 2");
    const ForestSpec &f = fa.spec;
    if (f.L < 2 || f.L > kMortonBits) return set_error(c, SV_ERR_INVALID, "forest leaf level %d", f.L);
    SV_TRY(fmm_state(c));
    Fmm &F = *c->fmm;
    SV_TRY(ensure_tables(c, F, p, fa.ws));
    F.trim = c->P.fmm_near == 2 && fa.ws == 2;
    if (!F.ftree) F.ftree = new Tree();
    SV_TRY(tree_forest_reserve(c, *F.ftree, f));
    const int NC = p * (p + 1) / 2;
    const int ns1 = 2 * fa.ws + 1, ns = ns1 * ns1 * ns1, cap = 7 * ns;
    auto rounded = [](size_t sz) { return (sz + 255) & ~(size_t)255; };
    size_t bytes = 0;
    for (int l = 0; l <= f.L; l++) {
        const size_t nb = (size_t)f.cap[l];
        F.fchunks[l] = m2l_chunks((int)nb);
        bytes += 2 * rounded(nb * NC * sizeof(float2)) + rounded(nb * ns * sizeof(int)) +
                 rounded(nb * cap * sizeof(int2)) + 2 * rounded(nb * sizeof(int));
        if (F.fchunks[l] > 1) bytes += rounded(nb * F.fchunks[l] * NC * sizeof(float2));
    }
    bytes += rounded((size_t)f.cap[f.L] * kFarDirectCap * sizeof(int)) + rounded((size_t)f.cap[f.L] * sizeof(int));
    const size_t item_bytes = near_items_room(f.n, f.cap[f.L]) * sizeof(int2);
    bytes += rounded(item_bytes);
    if (F.farena_bytes < bytes) {
        cudaFree(F.farena);
        F.farena = nullptr;
        F.farena_bytes = 0;
        SV_CK(c, cudaMalloc(&F.farena, bytes));
        F.farena_bytes = bytes;
    }
    char *q = (char *)F.farena;
    auto carve = [&](size_t sz) {
        char *r = q;
        q += (sz + 255) & ~(size_t)255;
        return (void *)r;
    };
    for (int l = 0; l <= kMortonBits; l++) {
        F.fM[l] = F.fL[l] = F.fpart[l] = nullptr;
        F.fnbr[l] = F.fcnt[l] = F.ftgt[l] = nullptr;
        F.flst[l] = nullptr;
    }
    for (int l = 0; l <= f.L; l++) {
        const size_t nb = (size_t)f.cap[l];
        F.fM[l] = (float2 *)carve(nb * NC * sizeof(float2));
        F.fL[l] = (float2 *)carve(nb * NC * sizeof(float2));
        F.fnbr[l] = (int *)carve(nb * ns * sizeof(int));
        F.flst[l] = (int2 *)carve(nb * cap * sizeof(int2));
        F.fcnt[l] = (int *)carve(nb * sizeof(int));
        F.ftgt[l] = (int *)carve(nb * sizeof(int));
        F.fpart[l] = F.fchunks[l] > 1 ? (float2 *)carve(nb * F.fchunks[l] * NC * sizeof(float2)) : F.fL[l];
    }
    F.ffd = (int *)carve((size_t)f.cap[f.L] * kFarDirectCap * sizeof(int));
    F.ffd_cnt = (int *)carve((size_t)f.cap[f.L] * sizeof(int));
    F.fitems = (int2 *)carve(item_bytes);
    if (c->P.fmm_m2l_tc >= 0 && f.L >= 2) {
        // room of the tensor-core M2L: the last run's translations with a
        // margin, at least 32 per box of the M2L levels (a graph keeps the
        // buffers' addresses, so the room only changes here, at plan time)
        int64_t boxes = 0;
        for (int l = 2; l <= f.L; l++) boxes += f.cap[l];
        const int64_t last = F.tc.h_ctl && F.tc.p == p && F.tc.ws == fa.ws ? F.tc.h_ctl[0] : 0;
        SV_TRY(m2l_tc_prepare(c, F.tc, p, fa.ws, std::max<int64_t>(last + last / 4, 32 * boxes)));
    }
    if (F.frel_cap < f.n) {
        cudaFree(F.frel);
        F.frel = nullptr;
        SV_CK(c, cudaMalloc(&F.frel, sizeof(float4) * (size_t)std::max(f.n, 1)));
        F.frel_cap = f.n;
    }
    return SV_OK;
}

sv_status fmm_forest_tc_grow(sv_ctx *c) {
    Fmm &F = *c->fmm;
    const int64_t need = F.tc.h_ctl ? F.tc.h_ctl[0] : 0;  // the true count of the run that overflowed
    // expanding plumes add ~25 % translations per step: four times the count
    // lasts ~6 steps; the room stays within 40 % of the device's memory
    // (beyond it the rotation kernel takes the translations that do not fit)
    size_t free_b = 0, total_b = 0;
    SV_CK(c, cudaMemGetInfo(&free_b, &total_b));
    const int p = F.tc.p;
    const double per_entry = 16.0 + (double)(((size_t)p * (p + 1) * 4 + 15) / 16 * 16);
    const int64_t limit = (int64_t)(0.4 * (double)total_b / per_entry);
    const int64_t want = std::min<int64_t>(4 * need, limit);
    if (want <= F.tc.cap) return SV_OK;
    return m2l_tc_prepare(c, F.tc, p, F.tc.ws, want, true);
}

bool fmm_forest_tc_used(const sv_ctx *c) {
    const Fmm *F = c->fmm;
    return F && F->tc.launched && F->tc.h_ctl && !F->tc.h_ctl[2];
}

bool fmm_forest_tc_overflowed(const sv_ctx *c) {
    const Fmm *F = c->fmm;
    return F && F->tc.launched && F->tc.h_ctl && F->tc.h_ctl[2];
}

__global__ void max_count_kernel(const int4 *__restrict__ coord, const int *__restrict__ nbd, int cap,
                                 int *__restrict__ out) {
    const int nb = level_boxes(cap, nbd);
    int m = 0;
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nb; b += gridDim.x * blockDim.x) m = max(m, coord[b].w);
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0 && m) atomicMax(out, m);
}

sv_status fmm_forest_max_leaf(sv_ctx *c, const ForestArgs &fa, int *out) {
    if (!c->fmm || !c->fmm->ftree) {
        *out = 0;
        return SV_OK;
    }
    const int L = fa.spec.L;
    int *d = nullptr;
    SV_CK(c, cudaMallocAsync(&d, sizeof(int), c->stream));
    SV_CK(c, cudaMemsetAsync(d, 0, sizeof(int), c->stream));
    max_count_kernel<<<forest_grid(fa.spec.cap[L], 256), 256, 0, c->stream>>>(c->fmm->ftree->lv[L].coord,
                                                                             fa.d_nbox + L, fa.spec.cap[L], d);
    SV_CK(c, cudaMemcpyAsync(c->h_scalar, d, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    SV_CK(c, cudaFreeAsync(d, c->stream));
    SV_CK(c, cudaStreamSynchronize(c->stream));
    memcpy(out, c->h_scalar, sizeof(int));
    return SV_OK;
}

sv_status fmm_forest_run(sv_ctx *c, const ForestArgs &fa) {
    if (fa.spec.n <= 0) return SV_OK;
    Fmm &F = *c->fmm;
    switch (fa.p) {
    case 4: return run_fmm_forest<4>(c, F, fa);
    case 6: return run_fmm_forest<6>(c, F, fa);
    case 8: return run_fmm_forest<8>(c, F, fa);
    default: return run_fmm_forest<10>(c, F, fa);
    }
}

sv_status fmm_counts(sv_ctx *c, double *m2l, double *pairs) {
    if (!c->fmm) {
        *m2l = *pairs = 0;
        return SV_OK;
    }
    SV_CK(c, cudaStreamSynchronize(c->stream));
    *m2l = (double)c->fmm->h_counts[0];
    *pairs = (double)c->fmm->h_counts[1];
    const M2LTc &tc = c->fmm->tc;
    c->stats.m2l_tc = tc.launched && tc.h_ctl && !tc.h_ctl[2];
    if (tc.launched && tc.h_ctl && tc.h_ctl[3])
        return set_error(c, SV_ERR_TIMEOUT, "tensor-core M2L: a bounded wait on the tensor cores gave up");
    return SV_OK;
}

}  // namespace sv
