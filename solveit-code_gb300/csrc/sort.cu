// sort.cu -- Morton ordering of the plume shared by every force method.
//
// The reference sorts particles by Morton index only inside the FMM
// (multipole_method_force_calculation.cpp:883-1083 presortMorton / sort /
// sortParticles, unsortParticles :1184).  Here every method works on a
// Morton-sorted copy so that consecutive targets are close in space; the
// caller's array order is untouched (results are scattered back), as the
// reference requires of updateAcceleration.
#include <cub/device/device_radix_sort.cuh>

#include <algorithm>
#include <cmath>
#include <utility>

#include "sv_internal.cuh"

namespace sv {
namespace {

constexpr int kRedThreads = 256;

__device__ __forceinline__ bool is_source(int32_t s) { return s == 1 || s == 2; }

constexpr double kBig = 1e300;  // bounds of an empty set

// Reduce (mn, mx) over a CTA of NT threads into threads 0..5 of the first
// warp: the value of axis d's minimum (thread d) or maximum (thread 3 + d).
template <int NT>
__device__ __forceinline__ long long block_bounds(long long (&mn)[3], long long (&mx)[3],
                                                  long long (&sh)[6][NT / 32]) {
#pragma unroll
    for (int d = 0; d < 3; d++) {
        for (int o = 16; o > 0; o >>= 1) {
            mn[d] = min(mn[d], __shfl_xor_sync(0xffffffffu, mn[d], o));
            mx[d] = max(mx[d], __shfl_xor_sync(0xffffffffu, mx[d], o));
        }
    }
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) {
        for (int d = 0; d < 3; d++) {
            sh[d][w] = mn[d];
            sh[3 + d][w] = mx[d];
        }
    }
    __syncthreads();
    long long v = 0;
    if (threadIdx.x < 6) {
        const int d = threadIdx.x;
        v = sh[d][0];
        for (int k = 1; k < NT / 32; k++) v = d < 3 ? min(v, sh[d][k]) : max(v, sh[d][k]);
    }
    return v;
}

// Root record from the bounds b[6] (min xyz, max xyz): origin (bbox min), cube
// side S = scale x the smallest power of two > the largest extent, with scale
// a multiple of 1/8 in [1, 2) (so every box side and every box-centre offset
// S/2^l * k, |k| < 8, is exact in binary floating point, FP32 included), bbox
// max, empty flag, and 2^21 / S for the keys.
__device__ __forceinline__ void write_root(double (&b)[6], double scale, double *__restrict__ root) {
    double ext = 0.0;
    const bool empty = b[0] > b[3];
    for (int d = 0; d < 3; d++) ext = fmax(ext, b[3 + d] - b[d]);
    if (empty) {
        for (int d = 0; d < 6; d++) b[d] = 0.0;
        ext = 0.0;
    }
    // guard against a zero extent (single particle) and keep the maximum
    // strictly inside the last cell: S > ext.
    double S = 1e-12;
    if (ext > 0.0) {
        int e;
        frexp(ext, &e);            // ext = f * 2^e, f in [0.5, 1)
        S = ldexp(1.0, e) * scale; // >= 2^e > ext
    }
    for (int d = 0; d < 3; d++) root[d] = b[d];
    root[3] = S;
    for (int d = 0; d < 3; d++) root[4 + d] = b[3 + d];
    root[7] = empty ? 1.0 : 0.0;
    root[8] = (double)(1u << kMortonBits) / S;
}

// Bounds of the source positions (status 1 or 2), exact: per-block minima and
// maxima, and the last block to finish reduces them and writes the root.  One
// launch on the integer pipe: a second kernel for the final reduction with
// FP64 minima took 8.2 us beside the partials' 4.3 (30,011 particles).
__global__ void __launch_bounds__(kRedThreads)
bbox_kernel(const double *__restrict__ x, const double *__restrict__ y, const double *__restrict__ z,
            const int32_t *__restrict__ st, int64_t n, long long *__restrict__ part, unsigned *__restrict__ done,
            double scale, double *__restrict__ root) {
    const long long lo0 = ordered_bits(__double_as_longlong(kBig)), hi0 = ordered_bits(__double_as_longlong(-kBig));
    __shared__ long long sh[6][kRedThreads / 32];
    __shared__ double bounds[6];
    __shared__ bool last;
    long long mn[3] = {lo0, lo0, lo0}, mx[3] = {hi0, hi0, hi0};
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        if (!is_source(st[i])) continue;
        const long long p[3] = {ordered_bits(__double_as_longlong(x[i])), ordered_bits(__double_as_longlong(y[i])),
                                ordered_bits(__double_as_longlong(z[i]))};
#pragma unroll
        for (int d = 0; d < 3; d++) {
            mn[d] = min(mn[d], p[d]);
            mx[d] = max(mx[d], p[d]);
        }
    }
    const long long v = block_bounds<kRedThreads>(mn, mx, sh);
    if (threadIdx.x < 6) part[blockIdx.x * 6 + threadIdx.x] = v;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int d = 0; d < 3; d++) {
        mn[d] = lo0;
        mx[d] = hi0;
    }
    for (int k = threadIdx.x; k < (int)gridDim.x; k += kRedThreads)
        for (int d = 0; d < 3; d++) {
            // a block whose bound is not a number is passed over, as fmin and fmax would
            const long long a = __ldcg(&part[k * 6 + d]), b = __ldcg(&part[k * 6 + 3 + d]);
            if (!ordered_nan(a)) mn[d] = min(mn[d], a);
            if (!ordered_nan(b)) mx[d] = max(mx[d], b);
        }
    const long long r = block_bounds<kRedThreads>(mn, mx, sh);
    if (threadIdx.x < 6) bounds[threadIdx.x] = __longlong_as_double(ordered_bits(r));
    __syncthreads();
    if (threadIdx.x == 0) {
        write_root(bounds, scale, root);
        root[14] = 0.0;  // both marks
        *done = 0;
    }
}

__device__ __forceinline__ uint64_t spread3(uint32_t v) { return morton_spread3(v); }

// Morton key of a source at (x, y, z); kInactiveKey for anything else.
__device__ __forceinline__ uint64_t morton_key(double x, double y, double z, int32_t st,
                                               const double *__restrict__ root) {
    if (!is_source(st)) return kInactiveKey;
    const double inv = root[8];  // 2^21 / S, exact (S is a power of two)
    const double p[3] = {x - root[0], y - root[1], z - root[2]};
    uint32_t c[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
        // floor(p * inv) clamped to [0, 2^21 - 1]: one round-down conversion
        // (PTX float-to-integer conversions saturate) and an integer clamp give
        // the same cell as floor, fmax and fmin in FP64, with half the FP64
        // operations of the key
        const int f = __double2int_rd(p[d] * inv);
        c[d] = (uint32_t)min(max(f, 0), (int)((1u << kMortonBits) - 1));
    }
    // bit order within a level: x lowest, then y, then z
    return spread3(c[0]) | (spread3(c[1]) << 1) | (spread3(c[2]) << 2);
}

__global__ void morton_keys(const double *__restrict__ x, const double *__restrict__ y,
                            const double *__restrict__ z, const int32_t *__restrict__ st,
                            int64_t n, const double *__restrict__ root,
                            uint64_t *__restrict__ keys, uint32_t *__restrict__ idx) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    idx[i] = (uint32_t)i;
    keys[i] = morton_key(x[i], y[i], z[i], st[i], root);
}

// The sorted copy's arrays and what its gather needs.
struct GatherArgs {
    const double *x, *y, *z, *q, *m, *qom;
    const int32_t *st;
    int64_t first, last;
    double kconst;
    double *xs, *ys, *zs;
    float *qs;
    double *qm;
    double *zax, *zay, *zaz;  // sorted accelerations to clear, or null
    float4 *ph, *pl, *pr;     // FP32 hi and lo positions and what they leave out to write, or null
    int abs_xy;               // ... relative to the z axis in x and y, not to the root's origin
    const double *root;
    int *marks;               // set with ph: [0] a source charge differs from particle 0's, [1] a source lies
                              // further than kWide from the origin of ph
};

// source charge of particle i (0: no source), and its K q / m (0: no target)
__device__ __forceinline__ float sorted_charge(const GatherArgs &a, uint32_t i) {
    return is_source(a.st[i]) ? (float)a.q[i] : 0.0f;
}
__device__ __forceinline__ double sorted_qm(const GatherArgs &a, uint32_t i) {
    const bool tgt = a.st[i] == 1 && (int64_t)i >= a.first && (int64_t)i < a.last && a.m[i] > 0.0;
    return tgt ? a.kconst * (a.qom ? a.qom[i] : a.q[i] / a.m[i]) : 0.0;
}

// Particle i into sorted slot s (every load before the first store); with ph, its marks as bits.
// A particle that is no source takes no part in any sum; it
// is put at the root's origin, for its own position may be anywhere and could become the
// origin of a block's FP32 coordinates (300 ions among as many lost ones within 100 m:
// 7.7e-7 against 1.2e-4 force error).
__device__ __forceinline__ int gather_one(const GatherArgs &a, const double *root, int64_t s, uint32_t i) {
    const bool src = is_source(a.st[i]);
    const double px = a.x[i], py = a.y[i], pz = a.z[i], k = sorted_qm(a, i);
    const double x = src ? px : root[0], y = src ? py : root[1], z = src ? pz : root[2];
    const float q = sorted_charge(a, i);
    a.xs[s] = x;
    a.ys[s] = y;
    a.zs[s] = z;
    a.qs[s] = q;
    a.qm[s] = k;
    if (a.zax) a.zax[s] = a.zay[s] = a.zaz[s] = 0.0;
    if (a.ph) {
        float4 h, l;
        split_hilo(x - (a.abs_xy ? 0.0 : root[0]), h.x, l.x);
        split_hilo(y - (a.abs_xy ? 0.0 : root[1]), h.y, l.y);
        split_hilo(z - root[2], h.z, l.z);
        h.w = q;
        l.w = k != 0.0 ? 1.f : 0.f;
        a.ph[s] = h;
        a.pl[s] = l;
        const bool wide = fmaxf(fabsf(h.x), fmaxf(fabsf(h.y), fabsf(h.z))) > kWide;
        float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
        if (wide)
            r = make_float4(split_rest(x, a.abs_xy ? 0.0 : root[0], h.x, l.x),
                            split_rest(y, a.abs_xy ? 0.0 : root[1], h.y, l.y), split_rest(z, root[2], h.z, l.z), 0.f);
        if (a.pr) a.pr[s] = r;
        return (h.w != sorted_charge(a, 0) ? 1 : 0) | (wide ? 2 : 0);
    }
    return 0;
}
__device__ __forceinline__ void set_marks(const GatherArgs &a, int bits) {
    if (bits & 1) a.marks[0] = 1;
    if (bits & 2) a.marks[1] = 1;
}

__global__ void gather_sorted(const uint32_t *__restrict__ idx, int64_t n, GatherArgs a) {
    const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (s < n) set_marks(a, gather_one(a, a.root, s, idx[s]));
}

// ------------------------------------------------------------- rank sort --
// Up to kRankSortMax particles are ordered by two launches instead of CUB's
// radix passes (one launch per 8 bits of the key, each a launch's latency at
// these sizes): chunks of CH particles are sorted in shared memory, then every
// particle's place in the whole order is its place in its own chunk plus its
// place in every other chunk (binary searches), and it is gathered there
// directly.  Both steps are stable, so the order is the one a stable radix
// sort of the same key bits gives.  Latency bound; the searches grow with
// n^2 / CH.  Serialised times of bounds, keys, order and gather, with CUB's
// nine passes and now: 256 particles 36 -> 8.8 us, 4,096 97 -> 24, 16,384
// 104 -> 35, 30,011 103 -> 45.  At 65,536 the searches take 83 us against the
// 54 of the six passes a tree needs, so the radix passes stay above
// kRankSortMax.
constexpr int64_t kRankSortMax = 32768;
constexpr int64_t kSmallChunkMax = 8192;  // chunks of 256 up to here, of 1024 above
constexpr int kOneChunk = 1024;           // one CTA sorts a plume of up to this many

// rank of `key` among the run v[0, len) of ascending keys: those below it, or
// (UPPER) not above it
template <bool UPPER>
__device__ __forceinline__ int run_rank(const uint64_t *__restrict__ v, int len, uint64_t key, int sh) {
    int lo = 0;
    for (int n = len; n > 0;) {
        const int half = n >> 1;
        const uint64_t k = v[lo + half] >> sh;
        const bool right = UPPER ? k <= key : k < key;
        lo = right ? lo + half + 1 : lo;
        n = right ? n - half - 1 : half;
    }
    return lo;
}

// Place of this thread's key in the sorted order of its chunk of CH
// threads' keys (bits sh and up; equal keys in thread order): by counting
// within the warp, then by doubling merges in shared memory.
template <int CH>
__device__ __forceinline__ int chunk_place(uint64_t key, int sh, uint64_t (*buf)[CH]) {
    const int lane = threadIdx.x & 31;
    const uint64_t mine = key >> sh;
    int r = 0;
#pragma unroll 8
    for (int k = 0; k < 32; k++) {
        const uint64_t o = __shfl_sync(0xffffffffu, mine, k);
        r += (o < mine || (o == mine && k < lane)) ? 1 : 0;
    }
    int pos = (threadIdx.x & ~31) + r, cur = 0;
    for (int run = 32; run < CH; run <<= 1, cur ^= 1) {
        buf[cur][pos] = mine;
        __syncthreads();
        const int start = pos & ~(run - 1), sib = start ^ run;
        const bool left = start < sib;
        const int o = left ? run_rank<false>(buf[cur] + sib, run, mine, 0) : run_rank<true>(buf[cur] + sib, run, mine, 0);
        pos = min(start, sib) + (pos - start) + o;
        // the next level writes the other buffer; this one is written again after its barrier
    }
    return pos;
}

// n <= CH: bounds, keys, order and gather in one CTA
template <int CH>
__global__ void __launch_bounds__(CH)
sort_one_chunk(int n, int sh, double scale, double *__restrict__ root, uint64_t *__restrict__ keys,
               uint32_t *__restrict__ idx, GatherArgs a) {
    __shared__ uint64_t buf[2][CH];
    __shared__ long long red[6][CH / 32];
    __shared__ double bounds[6];
    const int i = threadIdx.x;
    const long long lo0 = ordered_bits(__double_as_longlong(kBig)), hi0 = ordered_bits(__double_as_longlong(-kBig));
    long long mn[3] = {lo0, lo0, lo0}, mx[3] = {hi0, hi0, hi0};
    double p[3] = {0.0, 0.0, 0.0};
    int32_t st = 0;
    if (i < n) {
        st = a.st[i];
        p[0] = a.x[i];
        p[1] = a.y[i];
        p[2] = a.z[i];
        if (is_source(st))
#pragma unroll
            for (int d = 0; d < 3; d++) {
                const long long v = ordered_bits(__double_as_longlong(p[d]));
                if (!ordered_nan(v)) mn[d] = mx[d] = v;
            }
    }
    const long long v = block_bounds<CH>(mn, mx, red);
    if (i < 6) bounds[i] = __longlong_as_double(ordered_bits(v));
    __syncthreads();
    if (i == 0) {
        write_root(bounds, scale, root);
        root[14] = 0.0;  // both marks
    }
    __syncthreads();
    const uint64_t key = i < n ? morton_key(p[0], p[1], p[2], st, root) : kInactiveKey;
    const int pos = chunk_place<CH>(key, sh, buf);  // slots past n: inactive keys behind every particle
    if (i < n) {
        keys[pos] = key;
        idx[pos] = (uint32_t)i;
        set_marks(a, gather_one(a, root, pos, (uint32_t)i));
    }
}

// keys of a chunk of CH consecutive particles, sorted
template <int CH>
__global__ void __launch_bounds__(CH)
sort_chunks(int n, int sh, const double *__restrict__ root, uint64_t *__restrict__ ckeys,
            uint32_t *__restrict__ cidx, GatherArgs a) {
    __shared__ uint64_t buf[2][CH];
    const int base = blockIdx.x * CH, i = base + threadIdx.x;
    const uint64_t key = i < n ? morton_key(a.x[i], a.y[i], a.z[i], a.st[i], root) : kInactiveKey;
    const int pos = base + chunk_place<CH>(key, sh, buf);
    if (i < n) {
        ckeys[pos] = key;
        cidx[pos] = (uint32_t)i;
    }
}

// Sources first, otherwise in the caller's order, and the gather, in one launch:
// for the pair-once sums, which need no order among the sources (blocks that
// spread over the plume take the path that keeps the coordinates' parts below FP32
// for every tile).  Latency bound: one launch where the bounding box, the chunk sort
// and the ranks took three (25 us of 58 per evaluation at 4,096).  Every CTA counts the sources before its own particles itself,
// and takes the first source's position as the origin of the FP32 parts.
__global__ void __launch_bounds__(256)
sources_first(int n, uint32_t *__restrict__ idx, GatherArgs a, unsigned *__restrict__ done, int *__restrict__ bits) {
    __shared__ int wsum[8], tot[4];  // sources before this CTA, in all; first source; marks
    __shared__ double org[3];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    if (tid < 4) tot[tid] = tid == 2 ? n : 0;
    __syncthreads();
    int before = 0, all = 0, first = n;
#pragma unroll 4
    for (int c = 0; c < (int)gridDim.x; c++) {
        const int k = c * 256 + tid;
        if (k < n && is_source(a.st[k])) {
            all++;
            if (c < (int)blockIdx.x) before++;
            first = min(first, k);
        }
    }
    before = __reduce_add_sync(0xffffffffu, before);
    all = __reduce_add_sync(0xffffffffu, all);
    first = __reduce_min_sync(0xffffffffu, first);
    const int i = blockIdx.x * 256 + tid;
    const bool src = i < n && is_source(a.st[i]);
    const unsigned bal = __ballot_sync(0xffffffffu, src);
    if (lane == 0) {
        atomicAdd(&tot[0], before);
        atomicAdd(&tot[1], all);
        atomicMin(&tot[2], first);
        wsum[wid] = __popc(bal);
    }
    __syncthreads();
    if (tid < 3) org[tid] = tot[2] < n ? (tid == 0 ? a.x : tid == 1 ? a.y : a.z)[tot[2]] : 0.0;
    __syncthreads();
    int marks = 0;
    if (i < n) {
        int s = tot[0] + __popc(bal & ((1u << lane) - 1u));  // sources before this particle
        for (int w = 0; w < wid; w++) s += wsum[w];
        const int pos = src ? s : tot[1] + (i - s);
        idx[pos] = (uint32_t)i;
        marks = gather_one(a, org, pos, (uint32_t)i);
    }
    // the marks, from the last CTA to finish
    marks = __reduce_or_sync(0xffffffffu, marks);
    if (lane == 0 && marks) atomicOr(&tot[3], marks);
    __syncthreads();
    if (tid == 0) {
        if (tot[3]) atomicOr(bits, tot[3]);
        __threadfence();
        if (atomicAdd(done, 1u) == gridDim.x - 1) {
            const int b = atomicExch(bits, 0);
            a.marks[0] = b & 1;
            a.marks[1] = b >> 1;
            *done = 0;
        }
    }
}

// Every particle's rank over all chunks, and its gather: kRankLanes lanes per
// particle, each searching every kRankLanes-th chunk, their counts added; the
// lanes then move the particle's arrays side by side.  One lane per particle
// left a few warps per SM waiting for dependent loads (44 against 23 us at
// 30,011).
constexpr int kRankLanes = 8;
template <int CH>
__global__ void __launch_bounds__(256)
rank_gather(int n, int sh, const uint64_t *__restrict__ ckeys, const uint32_t *__restrict__ cidx,
            uint64_t *__restrict__ keys, uint32_t *__restrict__ idx, GatherArgs a) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int part = t % kRankLanes;
    const bool live = t / kRankLanes < n;
    const int s = live ? t / kRankLanes : n - 1;
    const uint64_t full = ckeys[s], key = full >> sh;
    const int own = s / CH, whole = n / CH;
    int rank = part == 0 ? s - own * CH : 0;
    // whole chunks two at a time, their searches independent of each other:
    // halving steps over CH keys.  Equal keys of earlier chunks count,
    // of later ones do not.
    auto below = [&](uint64_t k, bool eq) { return eq ? k <= key : k < key; };
    for (int c = part; c < whole; c += 2 * kRankLanes) {
        int lo[2] = {0, 0};
        const uint64_t *v[2];
        bool before[2];
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int cc = min(c + u * kRankLanes, whole - 1);
            v[u] = ckeys + (size_t)cc * CH;
            before[u] = cc < own;
        }
#pragma unroll
        for (int half = CH / 2; half > 0; half >>= 1)
#pragma unroll
            for (int u = 0; u < 2; u++)
                if (below(v[u][lo[u] + half - 1] >> sh, before[u])) lo[u] += half;
#pragma unroll
        for (int u = 0; u < 2; u++) {
            // CH - 1 keys are settled by the halving; the last one by itself
            if (below(v[u][lo[u]] >> sh, before[u])) lo[u]++;
            if (c + u * kRankLanes < whole && c + u * kRankLanes != own) rank += lo[u];
        }
    }
    // the short last chunk comes after this particle's own
    if (part == whole % kRankLanes && whole * CH < n && whole != own)
        rank += run_rank<false>(ckeys + (size_t)whole * CH, n - whole * CH, key, sh);
#pragma unroll
    for (int o = kRankLanes / 2; o > 0; o >>= 1) rank += __shfl_xor_sync(0xffffffffu, rank, o);
    if (!live) return;
    const uint32_t i = cidx[s];
    if (part < 3) {
        const double own = (part == 0 ? a.x : part == 1 ? a.y : a.z)[i];
        const double v = is_source(a.st[i]) ? own : a.root[part];  // as gather_one
        (part == 0 ? a.xs : part == 1 ? a.ys : a.zs)[rank] = v;
        if (a.ph) {
            float h, l;
            const double o = a.abs_xy && part < 2 ? 0.0 : a.root[part];
            split_hilo(v - o, h, l);
            if (a.pr) reinterpret_cast<float *>(a.pr + rank)[part] = fabsf(h) > kWide ? split_rest(v, o, h, l) : 0.f;
            reinterpret_cast<float *>(a.ph + rank)[part] = h;
            reinterpret_cast<float *>(a.pl + rank)[part] = l;
            if (fabsf(h) > kWide) a.marks[1] = 1;
        }
        return;
    }
    switch (part) {
    case 3: {
        const float q = sorted_charge(a, i);
        a.qs[rank] = q;
        if (a.ph) {
            a.ph[rank].w = q;
            if (q != sorted_charge(a, 0)) a.marks[0] = 1;
        }
        break;
    }
    case 4: {
        const double k = sorted_qm(a, i);
        a.qm[rank] = k;
        if (a.ph) a.pl[rank].w = k != 0.0 ? 1.f : 0.f;
        break;
    }
    case 5: keys[rank] = full; break;
    case 6: idx[rank] = i; break;
    default:
        if (a.zax) a.zax[rank] = a.zay[rank] = a.zaz[rank] = 0.0;
    }
}

// sorted slots of image copies (index >= n_orig) are sources only and have
// no place in the caller's arrays
__global__ void scatter_accel(const uint32_t *__restrict__ idx, int64_t n, int64_t n_orig,
                              const double *__restrict__ axs, const double *__restrict__ ays,
                              const double *__restrict__ azs, const double *__restrict__ far, int64_t fs,
                              const double *__restrict__ qm, int raw, double *__restrict__ ax,
                              double *__restrict__ ay, double *__restrict__ az) {
    const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (s >= n) return;
    const uint32_t i = idx[s];
    if ((int64_t)i >= n_orig) return;
    if (qm[s] == 0.0) {
        // not a target of this evaluation (status, range or mass): zero, whatever the
        // methods left in its sorted slot
        ax[i] = ay[i] = az[i] = 0.0;
    } else if (far) {
        ax[i] = axs[s] + far[s];
        ay[i] = ays[s] + far[fs + s];
        az[i] = azs[s] + far[2 * fs + s];
    } else if (raw) {
        const double k = qm[s];
        ax[i] = axs[s] * k;
        ay[i] = ays[s] * k;
        az[i] = azs[s] * k;
    } else {
        ax[i] = axs[s];
        ay[i] = ays[s];
        az[i] = azs[s];
    }
}

}  // namespace

sv_status ensure_sorted_capacity(sv_ctx *c, int64_t n) {
    Sorted &S = c->S;
    if (S.cap >= n && S.x) return SV_OK;
    cudaFree(S.x); cudaFree(S.y); cudaFree(S.z); cudaFree(S.q); cudaFree(S.qm);
    cudaFree(S.idx); cudaFree(S.keys); cudaFree(S.keys_alt); cudaFree(S.idx_alt);
    cudaFree(S.ax); cudaFree(S.ay); cudaFree(S.az); cudaFree(S.cub_tmp);
    cudaFree(S.root); cudaFree(S.red); cudaFree(S.ph); cudaFree(S.pl); cudaFree(S.pr);
    S = Sorted();
    const int64_t cap = n < 1024 ? 1024 : n;
    SV_CK(c, cudaMalloc(&S.x, cap * sizeof(double)));
    SV_CK(c, cudaMalloc(&S.y, cap * sizeof(double)));
    SV_CK(c, cudaMalloc(&S.z, cap * sizeof(double)));
    SV_CK(c, cudaMalloc(&S.q, cap * sizeof(float)));
    SV_CK(c, cudaMalloc(&S.qm, cap * sizeof(double)));
    SV_CK(c, cudaMalloc(&S.idx, cap * sizeof(uint32_t)));
    SV_CK(c, cudaMalloc(&S.idx_alt, cap * sizeof(uint32_t)));
    SV_CK(c, cudaMalloc(&S.keys, cap * sizeof(uint64_t)));
    SV_CK(c, cudaMalloc(&S.keys_alt, cap * sizeof(uint64_t)));
    SV_CK(c, cudaMalloc(&S.ax, cap * sizeof(double)));
    SV_CK(c, cudaMalloc(&S.ay, cap * sizeof(double)));
    SV_CK(c, cudaMalloc(&S.az, cap * sizeof(double)));
    size_t bytes = 0;
    cub::DoubleBuffer<uint64_t> kb(S.keys, S.keys_alt);
    cub::DoubleBuffer<uint32_t> vb(S.idx, S.idx_alt);
    SV_CK(c, cub::DeviceRadixSort::SortPairs(nullptr, bytes, kb, vb, (int)cap, 0, 64, c->stream));
    S.cub_bytes = bytes;
    SV_CK(c, cudaMalloc(&S.cub_tmp, bytes));
    S.red_blocks = 2 * device_sms();
    SV_CK(c, cudaMalloc(&S.red, (size_t)S.red_blocks * 6 * sizeof(long long)));
    SV_CK(c, cudaMalloc(&S.root, 16 * sizeof(double)));
    SV_CK(c, cudaMemsetAsync(S.root, 0, 16 * sizeof(double), c->stream));  // root[15]: bbox_kernel's block count
    S.cap = cap;
    return SV_OK;
}

// the FMM's root scale rounded down to a multiple of 1/8 (1 for the other methods)
static double root_scale(const sv_ctx *c) {
    const double s = c->P.fmm_root_scale;
    if (c->P.method != SV_METHOD_FMM || !(s >= 1.0)) return 1.0;
    return std::floor(std::min(s, 1.875) * 8.0) / 8.0;
}

sv_status sort_view(sv_ctx *c, const ParticleView &v, int64_t first, int64_t last) {
    const int64_t n = v.n;
    const SortWants want = std::exchange(c->S.want, SortWants());  // before the buffers are replaced
    SV_TRY(ensure_sorted_capacity(c, n));
    Sorted &S = c->S;
    S.raw = false;
    if (want.hilo && S.hl_cap < n) {
        cudaFree(S.ph);
        cudaFree(S.pl);
        S.ph = S.pl = nullptr;
        S.hl_cap = 0;
        SV_CK(c, cudaMalloc(&S.ph, sizeof(float4) * S.cap));
        SV_CK(c, cudaMalloc(&S.pl, sizeof(float4) * S.cap));
        S.hl_cap = S.cap;
    }
    if (want.rest && S.pr_cap < n) {
        cudaFree(S.pr);
        S.pr = nullptr;
        S.pr_cap = 0;
        SV_CK(c, cudaMalloc(&S.pr, sizeof(float4) * S.cap));
        S.pr_cap = S.cap;
    }
    S.n = n;
    S.n_orig = v.n_orig;
    // levels 1 .. levels occupy bits >= 3 (kMortonBits - levels); bit 63 marks inactive keys
    const int levels = std::max(1, std::min(kMortonBits, want.levels));
    S.key_levels = levels;
    const int sh = 3 * (kMortonBits - levels);
    GatherArgs ga{v.x, v.y, v.z, v.q, v.m, v.qom, v.status, first, std::min(last, v.n_orig), c->P.k_const,
                  S.x, S.y, S.z, S.q, S.qm, nullptr, nullptr, nullptr, want.hilo ? S.ph : nullptr,
                  want.hilo ? S.pl : nullptr, want.rest ? S.pr : nullptr, want.hl_abs ? 1 : 0, S.root, reinterpret_cast<int *>(S.root + 14)};
    if (want.zero) {
        ga.zax = S.ax;
        ga.zay = S.ay;
        ga.zaz = S.az;
    }
    if (want.any_order && n > 0) {
        sources_first<<<div_up(n, 256), 256, 0, c->stream>>>((int)n, S.idx, ga, reinterpret_cast<unsigned *>(S.root + 15),
                                                           reinterpret_cast<int *>(S.root + 13));
        SV_LAUNCHED(c);
        return SV_OK;
    }
    if (n <= kOneChunk) {
        if (n <= 256)
            sort_one_chunk<256><<<1, 256, 0, c->stream>>>((int)n, sh, root_scale(c), S.root, S.keys, S.idx, ga);
        else
            sort_one_chunk<kOneChunk><<<1, kOneChunk, 0, c->stream>>>((int)n, sh, root_scale(c), S.root, S.keys, S.idx,
                                                                      ga);
        SV_LAUNCHED(c);
        return SV_OK;
    }
    const int nb = div_up(n, 256);
    bbox_kernel<<<std::min(nb, S.red_blocks), kRedThreads, 0, c->stream>>>(
        v.x, v.y, v.z, v.status, n, S.red, reinterpret_cast<unsigned *>(S.root + 15), root_scale(c), S.root);
    SV_LAUNCHED(c);
    if (n <= kRankSortMax) {
        const int rgrid = div_up(n * kRankLanes, 256);
        if (n <= kSmallChunkMax) {
            sort_chunks<256><<<div_up(n, 256), 256, 0, c->stream>>>((int)n, sh, S.root, S.keys_alt, S.idx_alt, ga);
            SV_LAUNCHED(c);
            rank_gather<256><<<rgrid, 256, 0, c->stream>>>((int)n, sh, S.keys_alt, S.idx_alt, S.keys, S.idx, ga);
        } else {
            sort_chunks<1024><<<div_up(n, 1024), 1024, 0, c->stream>>>((int)n, sh, S.root, S.keys_alt, S.idx_alt, ga);
            SV_LAUNCHED(c);
            rank_gather<1024><<<rgrid, 256, 0, c->stream>>>((int)n, sh, S.keys_alt, S.idx_alt, S.keys, S.idx, ga);
        }
        SV_LAUNCHED(c);
        return SV_OK;
    }
    morton_keys<<<nb, 256, 0, c->stream>>>(v.x, v.y, v.z, v.status, n, S.root, S.keys, S.idx);
    SV_LAUNCHED(c);
    cub::DoubleBuffer<uint64_t> kb(S.keys, S.keys_alt);
    cub::DoubleBuffer<uint32_t> vb(S.idx, S.idx_alt);
    size_t bytes = S.cub_bytes;
    SV_CK(c, cub::DeviceRadixSort::SortPairs(S.cub_tmp, bytes, kb, vb, (int)n, sh, 3 * kMortonBits + 1, c->stream));
    c->launches += 2 * ((3 * levels + 1 + 7) / 8);  // CUB onesweep: histogram + passes
    if (kb.Current() != S.keys) {
        std::swap(S.keys, S.keys_alt);
    }
    if (vb.Current() != S.idx) {
        std::swap(S.idx, S.idx_alt);
    }
    gather_sorted<<<nb, 256, 0, c->stream>>>(S.idx, n, ga);
    SV_LAUNCHED(c);
    return SV_OK;
}

sv_status sort_state(sv_ctx *c, int64_t first, int64_t last) {
    const ParticleView v{c->x, c->y, c->z, c->q, c->m, force_status(c), c->n, c->n, c->qom};
    return sort_view(c, v, first, last);
}

sv_status unsort_accel(sv_ctx *c) {
    const int64_t n = c->S.n;
    scatter_accel<<<div_up(n, 256), 256, 0, c->stream>>>(c->S.idx, n, c->S.n_orig, c->S.ax, c->S.ay, c->S.az,
                                                         c->S.far, c->S.far_stride, c->S.qm, c->S.raw, c->ax, c->ay,
                                                         c->az);
    c->S.far = nullptr;
    c->S.raw = false;
    SV_LAUNCHED(c);
    return SV_OK;
}

}  // namespace sv
