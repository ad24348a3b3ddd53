// dm_sort.cuh -- spatial (Morton) ordering of a device-resident cloud.
//
// The all-pairs kernels test every pair, but their cost is decided per warp:
// a warp runs the precise path for a group of j as soon as ONE of its lanes'
// particles is within the cutoff.  With particles in input order a warp's
// particles are spread over the whole cloud and nearly every j group wakes
// it; in Morton order a warp's particles are a compact patch and only the j
// near that patch do.  The cloud therefore lives in Morton order on the
// device; `orig[s]` maps internal slot s back to the caller's particle index
// (used for the thermal RNG counter, for downloads and for the adaptive-dt
// pair pattern, all of which are defined on the caller's order).
//
// Sort: 24-bit Morton keys (12 bits per axis) and a deterministic, stable
// LSD radix sort with 8-bit digits (per-block digit histograms, a scan per
// digit, stable scatter ranked by a ballot-based digit match).  No atomics decide any
// order; the result depends only on the positions.
//
// The key box is the bounding box clipped to mean +- 4 standard deviations
// per axis.  A confined cloud that collapses and re-expands throws a few
// particles metres out while the rest stay within centimetres; over the
// plain bounding box a 12-bit cell is then wider than the cutoff and
// thousands of core particles share one key, so 32-particle groups are no
// longer compact.  Particles outside the clipped box take the edge cells.
#pragma once

#include <cooperative_groups.h>

#include "dm_device.cuh"

namespace dm {
namespace cg = cooperative_groups;

constexpr int kSortThreads = 256;
constexpr int kSortPerBlock = 4 * kSortThreads;  // keys per block
constexpr int kSortBits = 24;
constexpr int kSortDigitBits = 8;  // 24-bit keys: 3 passes
constexpr int kSortBuckets = 1 << kSortDigitBits;

// A sort that is due but not required (the cloud was sorted at most kOrderKeep
// steps ago and no upload has changed it) leaves a cloud alone whose order is
// still good: where the sweep is expected to look at less than kOrderSlack times
// what it would in the order as it was sorted, had the cloud since only grown or
// shrunk as a whole.  Expected from the boxes of the 32-particle groups: a
// box of w x h is looked at by the groups in (w + g) x (h + g) about it, g two
// cutoffs and a typical group's side.  Sides are capped at the cloud's size
// (a box cannot be looked at by more than all), and the size is one that single
// particles cannot move (block_order_record), so a particle thrown out counts as
// what it costs: its group is swept by every other.  Emulated on uniform disks
// of 4096, 16,384 and 262,144 particles, the ratio follows that of the pairs
// swept before and after a sort: particles that moved 0.2 mm each way 1.09
// (pairs 1.07-1.10), 1 mm 2.1 (2.5-3.0), 20 thrown out 2.2-2.5 (1.4-1.8), 400
// 15-24 (7-13).  Boxes against the distance between consecutive groups' centres,
// in the geometric mean, fell with every particle thrown: the uniform disk of
// 16,384, steps 5 to 24, swept 20.6% of all pairs and took 0.196 ms a step, now
// 16.7% and 0.184 ms; over 1500 steps 0.174 -> 0.164 ms.  A slack of 1 (always
// sorted) 0.193 and 0.167 ms, 1.05 0.185 and 0.166, 1.2 0.184 and 0.168, 1.4 0.186
// and 0.174; 262,144 particles 2.44 ms a step up to 1.1, 2.70 at 1.2.
// The check costs about 4 us of a 27 us sort (one cluster, latency bound):
// calm clouds of 4095 particles, 10 RK2 steps 594 -> 437 us, of 16,384 and 4 RK4
// steps 415 -> 345 us.
constexpr int kOrderKeep = 8;
constexpr float kOrderSlack = 1.1f;

// The order as last sorted.
struct OrderRecord {
    float area, sides;  // sums of w h and of w + h over the groups
    float scale;        // log2 of the cloud's size
    unsigned long long step;  // step index of the sort
};

// Whether a sort at step index `at` is less than kOrderKeep steps ago.  Counted
// from the sort on the device, so that the same state and the same steps are
// sorted at the same places whatever the cloud did before.
__device__ __forceinline__ bool order_is_recent(unsigned long long step, unsigned long long at) {
    return step - at < (unsigned long long)kOrderKeep;
}

// The sums of a and b over the block, in every thread; columns COL and COL + 1 of
// scratch (a row per warp) are free again after the block's next barrier.
template <int COL, int WARPS, int FIELDS>
__device__ __forceinline__ float2 block_sum2(float a, float b, float (&scratch)[WARPS][FIELDS]) {
    static_assert(FIELDS >= COL + 2, "two sums");
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    if ((threadIdx.x & 31) == 0) {
        scratch[threadIdx.x >> 5][COL] = a;
        scratch[threadIdx.x >> 5][COL + 1] = b;
    }
    __syncthreads();
    a = b = 0.0f;
#pragma unroll
    for (int w = 0; w < WARPS; w++) {
        a += scratch[w][COL];
        b += scratch[w][COL + 1];
    }
    return make_float2(a, b);
}

// The present order's record (but for the step): boxes gb, positions pa0 of
// `groups` groups; by every thread of the block.  The size is the geometric mean
// distance between the first particles of groups half the order apart: it does
// not change when particles mix, and one particle thrown out moves it only if
// it is such a first one, by its logarithm over their number.  Bound by two
// round trips to L2 and two block sums; each thread's first HELD boxes are on
// their way with the positions.
template <int HELD, int WARPS, int FIELDS>
__device__ __forceinline__ OrderRecord block_order_record(const float4 *gb, const float4 *pa0, int groups,
                                                          float (&scratch)[WARPS][FIELDS]) {
    constexpr int NT = 32 * WARPS;
    const int tid = threadIdx.x, half = groups >> 1;
    float4 held[HELD];
#pragma unroll
    for (int u = 0; u < HELD; u++)
        held[u] = (tid + u * NT < groups) ? __ldcg(gb + tid + u * NT) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float lg = 0.0f, cnt = 0.0f;
    const int g0 = tid * max(1, half / NT);  // a pair per thread is enough of a sample
    if (g0 < half) {
        const float4 a = __ldcg(pa0 + 32 * g0), b = __ldcg(pa0 + 32 * (g0 + half));
        const float dx = a.x - b.x, dy = a.y - b.y, d2 = fmaf(dx, dx, dy * dy);
        if (d2 > 0.0f && d2 < INFINITY) {  // NaN: neither
            lg = 0.5f * __log2f(d2);
            cnt = 1.0f;
        }
    }
    const float2 size = block_sum2<0>(lg, cnt, scratch);
    OrderRecord R;
    R.scale = size.x / fmaxf(size.y, 1.0f);
    const float cap = 2.0f * exp2f(R.scale);
    float area = 0.0f, sides = 0.0f;
    auto add = [&](const float4 &box) {
        const float w = fminf(box.z - box.x, cap), h = fminf(box.w - box.y, cap);  // NaN: cap
        area = fmaf(w, h, area);
        sides += w + h;
    };
#pragma unroll
    for (int u = 0; u < HELD; u++)
        if (tid + u * NT < groups) add(held[u]);
#pragma unroll HELD
    for (int g = tid + HELD * NT; g < groups; g += NT) add(__ldcg(gb + g));
    const float2 sum = block_sum2<2>(area, sides, scratch);
    __syncthreads();  // scratch is reused
    R.area = sum.x;
    R.sides = sum.y;
    R.step = 0;
    return R;
}

// Whether the order `now` is as good as it `was` (see kOrderSlack); false for NaN.
__device__ __forceinline__ bool order_is_good(const OrderRecord &now, const OrderRecord &was, int groups, float rc) {
    const float k = exp2f(now.scale - was.scale), G = (float)groups;
    const float g = 2.0f * rc + k * was.sides / (2.0f * G);
    return now.area + g * now.sides + G * g * g <= kOrderSlack * (k * k * was.area + k * g * was.sides + G * g * g);
}

constexpr int kMomentBlocks = 128;  // fixed partition of the moment reduction
constexpr int kMomentFields = 9;   // count, sum dx, sum dy, sum dx^2, sum dy^2, min x, min y, max x, max y

struct SortScratch {
    float *moments;            // [kMomentBlocks][kMomentFields] per-block partials
    double *box;               // [8]: key box x0, y0, extent; -; bounding box min x, min y, max x, max y
    OrderRecord *order;        // the cloud as last sorted (a batch: each cloud)
    int *keep;                 // set by order_check: the order is still good
    int *changed;              // number of the last upload that changed the state
    uint32_t *keys[2];
    int *vals[2];
    uint32_t *hist;            // [kSortBuckets * nblocks], then [kSortBuckets] totals
    double *stage[6];          // gather staging for x, y, vx, vy, q, m
    int *orig_stage;
};

// Moments of finite positions: count, sums of the offsets (dx, dy) from an
// origin and of their squares (the origin keeps the second moments well
// conditioned), and the bounding box.
struct Moments {
    double v[kMomentFields];
    __device__ __forceinline__ void clear() {
        for (int k = 0; k < 5; k++) v[k] = 0.0;
        v[5] = v[6] = INFINITY;
        v[7] = v[8] = -INFINITY;
    }
    __device__ __forceinline__ void add(double a, double b, double ox, double oy) {
        if (!(isfinite(a) && isfinite(b))) return;
        const double da = a - ox, db = b - oy;
        v[0] += 1.0;
        v[1] += da;
        v[2] += db;
        v[3] += da * da;
        v[4] += db * db;
        v[5] = fmin(v[5], a);
        v[6] = fmin(v[6], b);
        v[7] = fmax(v[7], a);
        v[8] = fmax(v[8], b);
    }
    __device__ __forceinline__ void merge(const double *o) {
        for (int k = 0; k < 5; k++) v[k] += o[k];
        v[5] = fmin(v[5], o[5]);
        v[6] = fmin(v[6], o[6]);
        v[7] = fmax(v[7], o[7]);
        v[8] = fmax(v[8], o[8]);
    }
    // butterfly over the warp; lane 0's result has a fixed evaluation order
    __device__ __forceinline__ void warp_reduce() {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            double o[kMomentFields];
#pragma unroll
            for (int k = 0; k < kMomentFields; k++) o[k] = __shfl_xor_sync(0xffffffffu, v[k], off);
            merge(o);
        }
    }
};

// Block-wide moments of positions i0, i0 + stride, ... < i1 (fixed
// partition and order: deterministic); the result is valid in thread 0.
__device__ __forceinline__ Moments block_moments(const double *__restrict__ x, const double *__restrict__ y,
                                                 int i0, int i1, int stride, double ox, double oy) {
    __shared__ double s[32][kMomentFields];
    Moments m;
    m.clear();
    for (int i = i0 + (int)threadIdx.x; i < i1; i += stride) m.add(x[i], y[i], ox, oy);
    m.warp_reduce();
    const int warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    if ((threadIdx.x & 31) == 0)
        for (int k = 0; k < kMomentFields; k++) s[warp][k] = m.v[k];
    __syncthreads();
    if (threadIdx.x == 0)
        for (int w = 1; w < nw; w++) m.merge(s[w]);
    __syncthreads();  // s is reused by the next call
    return m;
}

// Key box of a cloud from its moments: the bounding box clipped to mean +-
// 4 standard deviations per axis, as (x0, y0, extent); then the bounding
// box itself.  box[8]: x0, y0, extent, 0, min x, min y, max x, max y.
__device__ __forceinline__ void moments_to_box(const Moments &m, double ox, double oy, double *box) {
    double lo[2] = {0.0, 0.0}, hi[2] = {0.0, 0.0};
    const double n = m.v[0];
    if (n > 0.0) {
        const double org[2] = {ox, oy};
        for (int a = 0; a < 2; a++) {
            const double mean = m.v[1 + a] / n;
            const double sd = sqrt(fmax(m.v[3 + a] / n - mean * mean, 0.0));
            lo[a] = fmax(m.v[5 + a], org[a] + mean - 4.0 * sd);
            hi[a] = fmin(m.v[7 + a], org[a] + mean + 4.0 * sd);
            if (!(lo[a] <= hi[a])) {  // degenerate: fall back to the bounding box
                lo[a] = m.v[5 + a];
                hi[a] = m.v[7 + a];
            }
        }
    }
    box[0] = lo[0];
    box[1] = lo[1];
    box[2] = fmax(hi[0] - lo[0], hi[1] - lo[1]);
    box[3] = 0.0;
    for (int k = 0; k < 4; k++) box[4 + k] = (n > 0.0) ? m.v[5 + k] : 0.0;
}

__device__ __forceinline__ double finite_or_zero(double v) { return isfinite(v) ? v : 0.0; }

__device__ __forceinline__ void moments_f32_add(float *v, float4 a, float ox, float oy) {
    if (!(isfinite(a.x) && isfinite(a.y))) return;
    const float dx = a.x - ox, dy = a.y - oy;
    v[0] += 1.0f;
    v[1] += dx;
    v[2] += dy;
    v[3] = fmaf(dx, dx, v[3]);
    v[4] = fmaf(dy, dy, v[4]);
    v[5] = fminf(v[5], a.x);
    v[6] = fminf(v[6], a.y);
    v[7] = fmaxf(v[7], a.x);
    v[8] = fmaxf(v[8], a.y);
}

__device__ __forceinline__ void moments_f32_merge(float *v, const float *o) {
    for (int k = 0; k < 5; k++) v[k] += o[k];
    v[5] = fminf(v[5], o[5]);
    v[6] = fminf(v[6], o[6]);
    v[7] = fmaxf(v[7], o[7]);
    v[8] = fmaxf(v[8], o[8]);
}

// The block's moments of its threads' v; valid in thread 0.  scratch: a row per warp.
template <int WARPS, int FIELDS>
__device__ __forceinline__ void moments_f32_block(float (&v)[kMomentFields], float (&scratch)[WARPS][FIELDS]) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        float w[kMomentFields];
#pragma unroll
        for (int k = 0; k < kMomentFields; k++) w[k] = __shfl_xor_sync(0xffffffffu, v[k], o);
        moments_f32_merge(v, w);
    }
    if ((threadIdx.x & 31) == 0)
        for (int k = 0; k < kMomentFields; k++) scratch[threadIdx.x >> 5][k] = v[k];
    __syncthreads();
    if (threadIdx.x == 0)
        for (int w = 1; w < WARPS; w++) moments_f32_merge(v, scratch[w]);
}

// Key box of FP32 moments about the origin (ox, oy), as moments_to_box: x0, y0, extent.
__device__ __forceinline__ void key_box_f32(const float *v, float ox, float oy, float *box) {
    float lo[2] = {0.0f, 0.0f}, hi[2] = {0.0f, 0.0f};
    if (v[0] > 0.0f) {
        const float org[2] = {ox, oy};
        for (int a = 0; a < 2; a++) {
            const float mean = v[1 + a] / v[0];
            const float sd = sqrtf(fmaxf(v[3 + a] / v[0] - mean * mean, 0.0f));
            lo[a] = fmaxf(v[5 + a], org[a] + mean - 4.0f * sd);
            hi[a] = fminf(v[7 + a], org[a] + mean + 4.0f * sd);
            if (!(lo[a] <= hi[a])) {
                lo[a] = v[5 + a];
                hi[a] = v[7 + a];
            }
        }
    }
    box[0] = lo[0];
    box[1] = lo[1];
    box[2] = fmaxf(hi[0] - lo[0], hi[1] - lo[1]);
}

// Spreads the low 12 bits of v to the even bit positions.
__device__ __forceinline__ uint32_t spread_bits12(uint32_t v) {
    v &= 0x00000FFFu;
    v = (v | (v << 8)) & 0x00FF00FFu;
    v = (v | (v << 4)) & 0x0F0F0F0Fu;
    v = (v | (v << 2)) & 0x33333333u;
    v = (v | (v << 1)) & 0x55555555u;
    return v;
}

// Lanes of the warp holding the same 8-bit digit as this one, among the
// lanes with `valid` set: one ballot per digit bit.  Eight ballots cost far
// less than __match_any_sync when 32 warps of one block issue them (the
// match unit's throughput, not the ballots', bounds a one-block sort).
__device__ __forceinline__ uint32_t match_digit8(uint32_t d, bool valid) {
    uint32_t m = __ballot_sync(0xffffffffu, valid);
#pragma unroll
    for (int b = 0; b < kSortDigitBits; b++) {
        const bool bit = (d >> b) & 1u;
        const uint32_t bal = __ballot_sync(0xffffffffu, bit);
        m &= bit ? bal : ~bal;
    }
    return m;
}

// 24-bit Morton key of position (x, y) in a key box.
__device__ __forceinline__ uint32_t morton_key_f32(float x, float y, const float *box) {
    const float ext = box[2];
    const float scale = (ext > 0.0f && isfinite(ext)) ? 4095.0f / ext : 0.0f;
    const float fx = (x - box[0]) * scale, fy = (y - box[1]) * scale;
    const uint32_t qx = (fx > 0.0f) ? (uint32_t)fminf(fx, 4095.0f) : 0u;  // NaN: 0
    const uint32_t qy = (fy > 0.0f) ? (uint32_t)fminf(fy, 4095.0f) : 0u;
    return spread_bits12(qx) | (spread_bits12(qy) << 1);
}

// Position set 1 (see write_midpoint) of slot s and its group's box; whole warps.
__device__ __forceinline__ void write_midpoint_group(const CloudDev &c, int s, bool live, float4 *gbox, bool store,
                                                     double dt) {
    float4 A = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (live) {
        write_midpoint(c, s, c.x[s], c.y[s], c.vx[s], c.vy[s], dt);
        A = c.pa[1][s];
    }
    store_group_box(gbox, live, A.x, A.y, store);
}

// ---------------------------------------------------------------------------
// The sort of clouds larger than one cluster holds: order_check, sort_moments,
// sort_keys (with the first digit's histogram), per 8-bit digit radix_scan and
// radix_scatter (and radix_hist before the next), permute_gather,
// permute_commit and order_record.  Where order_check found the order still good the others
// return at once (`keep`; null: always sort).  Bound by launch latency and by
// a pass over the keys each (262,144 particles: ~60 us sorted, 17 us kept;
// with FP64 moments and keys, one block scanning all the counts and separate
// position and midpoint launches it took 150 us, every step).  The key box and
// the keys are FP32 functions of the positions' hi parts, as in sort_cluster.
// ---------------------------------------------------------------------------

__device__ __forceinline__ bool order_is_kept(const int *keep) { return keep && *keep; }

// One block: whether the cloud's order is still good (slot: of the step counter) ...
static __global__ void __launch_bounds__(1024) order_check(CloudDev c, SortScratch z, int slot, int upload) {
    pdl_wait();
    __shared__ float s[32][4];
    const int groups = (c.n + 31) / 32;
    const OrderRecord was = *z.order;  // on their way with the boxes
    const unsigned long long step = c.step_ctr[slot];
    const int changed = *z.changed;
    const OrderRecord now = block_order_record<8>(c.gbox[0], c.pa[0], groups, s);
    if (threadIdx.x == 0)
        *z.keep = order_is_good(now, was, groups, sqrtf(c.rc2_up)) && order_is_recent(step, was.step) &&
                  (upload == 0 || changed != upload);
}

// ... and, after a sort, how good it is.
static __global__ void __launch_bounds__(1024) order_record(CloudDev c, SortScratch z, int slot, const int *keep) {
    pdl_wait();
    if (order_is_kept(keep)) return;
    __shared__ float s[32][4];
    OrderRecord now = block_order_record<8>(c.gbox[0], c.pa[0], (c.n + 31) / 32, s);
    now.step = c.step_ctr[slot];
    if (threadIdx.x == 0) *z.order = now;
}

// Per-block moments of the cloud's positions (origin: its first particle).
static __global__ void __launch_bounds__(256) sort_moments(const float4 *__restrict__ pa0, int n, float *part,
                                                           const int *keep) {
    pdl_wait();
    if (order_is_kept(keep)) return;
    __shared__ float s[8][kMomentFields];
    const float4 p0 = pa0[0];
    const float ox = isfinite(p0.x) ? p0.x : 0.0f, oy = isfinite(p0.y) ? p0.y : 0.0f;
    float v[kMomentFields] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, INFINITY, INFINITY, -INFINITY, -INFINITY};
#pragma unroll 4
    for (int i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) moments_f32_add(v, pa0[i], ox, oy);
    moments_f32_block<8>(v, s);
    if (threadIdx.x == 0)
        for (int k = 0; k < kMomentFields; k++) part[blockIdx.x * kMomentFields + k] = v[k];
}

// The key box from the nparts blocks' moments (every block the same; block 0
// stores it), the keys of the block's kSortPerBlock particles and their first
// digit's histogram.
static __global__ void __launch_bounds__(kSortThreads) sort_keys(const float4 *__restrict__ pa0, int n, int nparts,
                                                                 SortScratch z, const int *keep) {
    pdl_wait();
    if (order_is_kept(keep)) return;
    __shared__ float box[3];
    __shared__ uint32_t h[kSortBuckets];
    h[threadIdx.x] = 0u;
    if (threadIdx.x < 32) {
        float v[kMomentFields] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, INFINITY, INFINITY, -INFINITY, -INFINITY};
        for (int b = threadIdx.x; b < nparts; b += 32) moments_f32_merge(v, z.moments + b * kMomentFields);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            float w[kMomentFields];
#pragma unroll
            for (int k = 0; k < kMomentFields; k++) w[k] = __shfl_xor_sync(0xffffffffu, v[k], o);
            moments_f32_merge(v, w);
        }
        if (threadIdx.x == 0) {
            const float4 p0 = pa0[0];
            key_box_f32(v, isfinite(p0.x) ? p0.x : 0.0f, isfinite(p0.y) ? p0.y : 0.0f, box);
            if (blockIdx.x == 0) {
                for (int k = 0; k < 3; k++) z.box[k] = box[k];
                z.box[3] = 0.0;
                for (int k = 0; k < 4; k++) z.box[4 + k] = (v[0] > 0.0f) ? (double)v[5 + k] : 0.0;
            }
        }
    }
    __syncthreads();
    for (int k = 0; k < 4; k++) {
        const int e = blockIdx.x * kSortPerBlock + k * kSortThreads + threadIdx.x;
        if (e >= n) continue;
        const float4 p = pa0[e];
        const uint32_t key = morton_key_f32(p.x, p.y, box);
        z.keys[0][e] = key;
        z.vals[0][e] = e;
        atomicAdd(&h[key & (kSortBuckets - 1)], 1u);
    }
    __syncthreads();
    z.hist[threadIdx.x * gridDim.x + blockIdx.x] = h[threadIdx.x];
}

static __global__ void __launch_bounds__(kSortThreads) radix_hist(const uint32_t *__restrict__ keys, int n,
                                                                  int shift, uint32_t *hist, const int *keep) {
    pdl_wait();
    if (order_is_kept(keep)) return;
    __shared__ uint32_t h[kSortBuckets];
    h[threadIdx.x] = 0u;
    __syncthreads();
    for (int k = 0; k < 4; k++) {
        const int e = blockIdx.x * kSortPerBlock + k * kSortThreads + threadIdx.x;
        if (e < n) atomicAdd(&h[(keys[e] >> shift) & (kSortBuckets - 1)], 1u);
    }
    __syncthreads();
    hist[threadIdx.x * gridDim.x + blockIdx.x] = h[threadIdx.x];
}

// Exclusive prefix over the block of 256 threads; total: the block's sum.
__device__ __forceinline__ uint32_t block_exclusive_256(uint32_t v, uint32_t &total) {
    __shared__ uint32_t ws[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) ws[warp] = inc;
    __syncthreads();
    uint32_t before = 0u;
    total = 0u;
    for (int w = 0; w < 8; w++) {
        before += (w < warp) ? ws[w] : 0u;
        total += ws[w];
    }
    __syncthreads();
    return before + inc - v;
}

// Block d: the exclusive prefix of digit d's nblocks counts, in place, and
// their total (hist[kSortBuckets * nblocks + d]).  The digits' own bases are
// formed by radix_scatter's blocks.  (One block over all the counts took 21 us
// for the 65,536 of a 262,144-particle sort.)
static __global__ void __launch_bounds__(256) radix_scan(uint32_t *hist, int nblocks, const int *keep) {
    pdl_wait();
    if (order_is_kept(keep)) return;
    uint32_t *row = hist + (size_t)blockIdx.x * nblocks, carry = 0u;
    for (int b0 = 0; b0 < nblocks; b0 += 256) {
        const int b = b0 + threadIdx.x;
        uint32_t total;
        const uint32_t pre = block_exclusive_256((b < nblocks) ? row[b] : 0u, total);
        if (b < nblocks) row[b] = carry + pre;
        carry += total;
    }
    if (threadIdx.x == 0) hist[(size_t)kSortBuckets * nblocks + blockIdx.x] = carry;
}

// Stable scatter: elements are ranked in index order (chunk, warp, lane).
static __global__ void __launch_bounds__(kSortThreads) radix_scatter(
    const uint32_t *__restrict__ kin, const int *__restrict__ vin, uint32_t *kout, int *vout, int n,
    int shift, const uint32_t *__restrict__ hist, const int *keep) {
    pdl_wait();
    if (order_is_kept(keep)) return;
    constexpr int NWARP = kSortThreads / 32;
    static_assert(kSortThreads == kSortBuckets, "a thread per digit");
    __shared__ uint32_t base[kSortBuckets];
    __shared__ uint32_t wcnt[NWARP][kSortBuckets];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    {
        uint32_t all;
        const uint32_t first = block_exclusive_256(hist[(size_t)kSortBuckets * gridDim.x + threadIdx.x], all);
        base[threadIdx.x] = first + hist[(size_t)threadIdx.x * gridDim.x + blockIdx.x];
    }
    for (int k = 0; k < 4; k++) {
        for (int e = threadIdx.x; e < NWARP * kSortBuckets; e += kSortThreads) (&wcnt[0][0])[e] = 0u;
        __syncthreads();
        const int e = blockIdx.x * kSortPerBlock + k * kSortThreads + threadIdx.x;
        const bool valid = e < n;
        const uint32_t key = valid ? kin[e] : 0u;
        const int d = (int)((key >> shift) & (kSortBuckets - 1));
        const uint32_t peers = match_digit8((uint32_t)d, valid);
        const uint32_t rank = __popc(peers & ((1u << lane) - 1u));
        if (valid && rank == 0) wcnt[warp][d] = __popc(peers);
        __syncthreads();
        if (valid) {
            uint32_t pos = base[d] + rank;
            for (int w = 0; w < warp; w++) pos += wcnt[w][d];
            kout[pos] = key;
            vout[pos] = vin[e];
        }
        __syncthreads();
        uint32_t add = 0;
        for (int w = 0; w < NWARP; w++) add += wcnt[w][threadIdx.x];
        base[threadIdx.x] += add;
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// One-launch sort for clouds of up to kSmallSortMax particles: a cluster of
// CTAS blocks, block r owning sorted positions [r*P, (r+1)*P),
// P = kSmallSortMax / CTAS.  Key box, keys, the three 8-bit LSD
// passes and the gather of the cloud's arrays in the new order run in one
// launch: per pass each block counts its digits per warp, the blocks'
// digit totals meet through distributed shared memory, and every element is
// stored straight into the shared memory of the block owning its new
// position.  The multi-kernel path above needs twelve dependent launches
// for it; a single block was no better (one SM's issue rate).
//
// Element order: block r, warp w, round k, lane l is element
// r*P + w*32*R + k*32 + l (R = P / threads).  Digits are ranked in that order
// (lanes with equal digits found by match_digit8) and bases are laid out
// digit-major over (digit, block, warp), so the sort is stable and depends
// only on the positions.  The key
// box and keys are FP32 functions of the positions' hi parts: GB300's FP64
// rate (~2 FMA per clock per SM) would dominate a pass over 16384 doubles,
// and any order is correct (the permutation moves every array together).
// ---------------------------------------------------------------------------
constexpr int kSmallSortMax = 16384;
constexpr int kErrSortPermutation = 8;  // error bit: the cluster sort's ranks were inconsistent
constexpr int kSortClusterThreads = 512;
constexpr int kSortClusterWarps = kSortClusterThreads / 32;

// CTAS blocks of PER elements, ROUNDS per thread: 8 (a portable cluster) or
// 16 (non-portable; half the elements per SM)
template <int CTAS>
struct SortClusterShape {
    static constexpr int per = kSmallSortMax / CTAS;
    static constexpr int rounds = per / kSortClusterThreads;
    static_assert(rounds * kSortClusterThreads == per, "whole rounds per thread");
};

template <int CTAS>
struct SortClusterSmem {
    static constexpr int kPer = SortClusterShape<CTAS>::per;
    uint32_t keys[2][kPer];
    uint16_t slot[2][kPer];
    uint32_t wcnt[kSortClusterWarps][kSortBuckets];  // per-warp digit counts, then offsets within the block
    uint32_t ctot[kSortBuckets];      // this block's digit totals (read by the whole cluster)
    uint32_t dbase[kSortBuckets];     // first sorted position of (digit, this block)
    uint32_t part[kSortBuckets / 32];
    float wmom[kSortClusterWarps][kMomentFields];
    float mom[kMomentFields];  // this block's moments (read by the whole cluster)
    float box[3];
};
template <int CTAS>
constexpr size_t sort_cluster_smem() { return sizeof(SortClusterSmem<CTAS>); }

// pa0: the FP32 hi parts of the current positions (position set 0 holds them
// at every step boundary).  The cloud's x, y, vx, vy, q, m and orig end up in
// the new order, with position set 0, set 1 for time step dt (if mid) and
// their group boxes rewritten.  Without `force` (or an upload of number
// `upload` that changed the state) a cloud in good order (see kOrderKeep) is
// left as it is; if `mid` and not `mid_ready` its set 1 is
// written.  slot: of the step counter.  Launched as one cluster of CTAS blocks.
template <int CTAS>
static __global__ void __launch_bounds__(kSortClusterThreads, 1)
    sort_cluster(const float4 *__restrict__ pa0, CloudDev c, SortScratch z, double dt, bool mid, bool mid_ready,
                 bool force, int slot, int upload) {
    constexpr int kSortClusterCtas = CTAS;
    constexpr int kSortClusterPer = SortClusterShape<CTAS>::per;
    constexpr int kSortClusterRounds = SortClusterShape<CTAS>::rounds;
    pdl_wait();
    extern __shared__ __align__(128) unsigned char smem_raw[];
    SortClusterSmem<CTAS> &S = *reinterpret_cast<SortClusterSmem<CTAS> *>(smem_raw);
    cg::cluster_group cl = cg::this_cluster();
    const int r = (int)cl.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n = c.n;
    const int e0 = r * kSortClusterPer;
    const int groups = (n + 31) / 32;

    // every block comes to the same decision
    if (!force && (upload == 0 || *z.changed != upload)) {
        const OrderRecord was = *z.order;  // on their way with the boxes
        const unsigned long long step = c.step_ctr[slot];
        const OrderRecord now = block_order_record<1>(c.gbox[0], pa0, groups, S.wmom);
        if (order_is_good(now, was, groups, sqrtf(c.rc2_up)) && order_is_recent(step, was.step)) {
            if (mid && !mid_ready)
                for (int k = 0; k < kSortClusterRounds; k++) {
                    const int s = e0 + k * kSortClusterThreads + tid;
                    write_midpoint_group(c, s, s < n, c.gbox[1] + (s >> 5), (s & ~31) < c.n_pad, dt);
                }
            return;
        }
    }

    // this block's positions, loaded once (moments, then keys)
    float4 pos[kSortClusterRounds];
#pragma unroll
    for (int k = 0; k < kSortClusterRounds; k++) {
        const int e = e0 + k * kSortClusterThreads + tid;
        pos[k] = (e < n) ? pa0[e] : make_float4(NAN, NAN, 0.0f, 0.0f);
    }
    // moments of this block's slice, then of the cloud: lanes 0..CTAS-1 of warp 0
    // fetch the cluster's blocks' moments and merge them in a fixed butterfly
    // (commutative steps), so every block derives the same key box
    const float4 p0 = pa0[0];
    const float ox = isfinite(p0.x) ? p0.x : 0.0f, oy = isfinite(p0.y) ? p0.y : 0.0f;
    {
        float v[kMomentFields] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, INFINITY, INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int k = 0; k < kSortClusterRounds; k++) moments_f32_add(v, pos[k], ox, oy);
        moments_f32_block<kSortClusterWarps>(v, S.wmom);
        if (tid == 0)
            for (int k = 0; k < kMomentFields; k++) S.mom[k] = v[k];
    }
    cl.sync();
    if (warp == 0) {
        float v[kMomentFields];
        const float *mb = cl.map_shared_rank(S.mom, lane & (kSortClusterCtas - 1));
#pragma unroll
        for (int k = 0; k < kMomentFields; k++) v[k] = mb[k];
#pragma unroll
        for (int off = 1; off < kSortClusterCtas; off <<= 1) {
            float o[kMomentFields];
#pragma unroll
            for (int k = 0; k < kMomentFields; k++) o[k] = __shfl_xor_sync(0xffffffffu, v[k], off);
            moments_f32_merge(v, o);
        }
        if (lane == 0) {
            key_box_f32(v, ox, oy, S.box);
            if (r == 0) {  // the key box and the bounding box, as the multi-kernel path writes them
                z.box[0] = S.box[0];
                z.box[1] = S.box[1];
                z.box[2] = S.box[2];
                z.box[3] = 0.0;
                for (int k = 0; k < 4; k++) z.box[4 + k] = (v[0] > 0.0f) ? (double)v[5 + k] : 0.0;
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kSortClusterRounds; k++) {
        const int li = k * kSortClusterThreads + tid, e = e0 + li;
        S.keys[0][li] = (e < n) ? morton_key_f32(pos[k].x, pos[k].y, S.box) : 0u;
        S.slot[0][li] = (uint16_t)e;
    }
    __syncthreads();

    const uint32_t lower = (1u << lane) - 1u;
    int cur = 0;
    for (int shift = 0; shift < kSortBits; shift += kSortDigitBits) {
        for (int d = lane; d < kSortBuckets; d += 32) S.wcnt[warp][d] = 0u;
        __syncwarp();
        uint32_t dk[kSortClusterRounds], rk[kSortClusterRounds];
#pragma unroll
        for (int k = 0; k < kSortClusterRounds; k++) {
            const int li = warp * (32 * kSortClusterRounds) + k * 32 + lane;
            const bool valid = e0 + li < n;
            const uint32_t d = (S.keys[cur][li] >> shift) & (kSortBuckets - 1);
            const uint32_t peers = match_digit8(d, valid);
            rk[k] = S.wcnt[warp][d] + __popc(peers & lower);  // rank within the warp
            dk[k] = valid ? d : kSortBuckets;
            __syncwarp();
            if (valid && (peers & lower) == 0u) S.wcnt[warp][d] += __popc(peers);
            __syncwarp();
        }
        __syncthreads();
        if (tid < kSortBuckets) {  // per digit: offsets of the warps, block total
            uint32_t run = 0u;
            for (int w = 0; w < kSortClusterWarps; w++) {
                const uint32_t v = S.wcnt[w][tid];
                S.wcnt[w][tid] = run;
                run += v;
            }
            S.ctot[tid] = run;
        }
        cl.sync();  // every block's totals are complete
        uint32_t tot = 0u, pre = 0u, inc = 0u;
        if (tid < kSortBuckets) {
            for (int b = 0; b < kSortClusterCtas; b++) {
                const uint32_t v = *cl.map_shared_rank(&S.ctot[tid], b);
                tot += v;
                pre += (b < r) ? v : 0u;
            }
            inc = tot;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, inc, off);
                if (lane >= off) inc += v;
            }
            if (lane == 31) S.part[warp] = inc;
        }
        __syncthreads();
        if (tid < kSortBuckets) {
            uint32_t wb = 0u;
            for (int w = 0; w < warp; w++) wb += S.part[w];
            S.dbase[tid] = wb + inc - tot + pre;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kSortClusterRounds; k++) {
            if (dk[k] < (uint32_t)kSortBuckets) {
                const int li = warp * (32 * kSortClusterRounds) + k * 32 + lane;
                const uint32_t pos = S.dbase[dk[k]] + S.wcnt[warp][dk[k]] + rk[k];
                if (pos >= (uint32_t)n) {  // cannot happen for a consistent count; never store out of range
                    atomicOr(c.err, kErrSortPermutation);
                    continue;
                }
                const int dst = (int)(pos / kSortClusterPer), off = (int)(pos % kSortClusterPer);
                *cl.map_shared_rank(&S.keys[cur ^ 1][off], dst) = S.keys[cur][li];
                *cl.map_shared_rank(&S.slot[cur ^ 1][off], dst) = S.slot[cur][li];
            }
        }
        cl.sync();  // all elements placed; all remote reads of this pass done
        cur ^= 1;
    }

    // gather: new slot s takes old slot S.slot[cur][s - e0]; plain loads (the
    // arrays are overwritten in place below), all issued before any store
    int src[kSortClusterRounds];
#pragma unroll
    for (int k = 0; k < kSortClusterRounds; k++) {
        const int li = k * kSortClusterThreads + tid, s = e0 + li;
        int o = (s < n) ? (int)S.slot[cur][li] : 0;
        if (s < n && o >= n) {  // as above: flag and keep the slot rather than read out of range
            atomicOr(c.err, kErrSortPermutation);
            o = s;
        }
        src[k] = o;
    }
    const double *in[7] = {c.x, c.y, c.vx, c.vy, c.q, c.m, c.invm};
    double val[7][kSortClusterRounds];
    int ov[kSortClusterRounds];
#pragma unroll
    for (int k = 0; k < kSortClusterRounds; k++) {
        const bool ok = e0 + k * kSortClusterThreads + tid < n;
#pragma unroll
        for (int a = 0; a < 7; a++) val[a][k] = ok ? in[a][src[k]] : 0.0;
        ov[k] = ok ? c.orig[src[k]] : 0;
    }
    // Every block of the cluster holds its sources in registers, and the
    // cluster barrier orders those loads before any block's stores.  The
    // cluster covers every slot of the cloud, so the cloud's arrays are
    // rewritten in place in the new order, with position sets 0 and 1 (the
    // next pass's inputs), the padding slots and the 32-particle group boxes.
    cl.sync();
#pragma unroll
    for (int k = 0; k < kSortClusterRounds; k++) {
        const int s = e0 + k * kSortClusterThreads + tid;  // a warp holds 32 consecutive slots
        float2 h[2] = {};
        if (s < n) {
            const double x = val[0][k], y = val[1][k];
            c.vx[s] = val[2][k];
            c.vy[s] = val[3][k];
            c.q[s] = val[4][k];
            c.m[s] = val[5][k];
            c.invm[s] = val[6][k];
            c.orig[s] = ov[k];
            write_stage_position(c, 0, s, x, y);  // set 0 is the state: x, y
            h[0] = make_float2(__double2float_rn(x), __double2float_rn(y));
            if (mid) {
                write_midpoint(c, s, x, y, val[2][k], val[3][k], dt);
                const float4 A = c.pa[1][s];
                h[1] = make_float2(A.x, A.y);
            }
        } else if (s < c.n_pad) {
            write_padding(c, s);
            c.q[s] = 0.0;
            c.m[s] = 1.0;
        }
        store_group_box(c.gbox[0] + (s >> 5), s < n, h[0].x, h[0].y, (s & ~31) < c.n_pad);
        if (mid) store_group_box(c.gbox[1] + (s >> 5), s < n, h[1].x, h[1].y, (s & ~31) < c.n_pad);
    }
    cl.sync();  // the boxes are written (ordered at cluster scope)
    if (r == 0) {
        OrderRecord now = block_order_record<1>(c.gbox[0], c.pa[0], groups, S.wmom);
        now.step = c.step_ctr[slot];
        if (tid == 0) *z.order = now;
    }
}

// new slot s takes old slot perm[s]: gather into staging ...
static __global__ void permute_gather(CloudDev c, const int *__restrict__ perm, SortScratch z, const int *keep) {
    pdl_wait();
    if (order_is_kept(keep)) return;
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= c.n) return;
    const int o = perm[s];
    z.stage[0][s] = c.x[o];
    z.stage[1][s] = c.y[o];
    z.stage[2][s] = c.vx[o];
    z.stage[3][s] = c.vy[o];
    z.stage[4][s] = c.q[o];
    z.stage[5][s] = c.m[o];
    z.orig_stage[s] = c.orig[o];
}

// ... and copy back (the cloud's array addresses never change, so captured
// CUDA graphs stay valid), with position set 0, set 1 for time step dt (if
// mid), the padding and the group boxes.  Blocks of 256.
static __global__ void __launch_bounds__(256) permute_commit(CloudDev c, SortScratch z, double dt, bool mid,
                                                             bool mid_ready, const int *keep) {
    pdl_wait();
    const int s = blockIdx.x * 256 + threadIdx.x;  // n_pad: whole warps
    const bool live = s < c.n, store = s < c.n_pad;
    if (!order_is_kept(keep)) {
        float xh = 0.0f, yh = 0.0f;
        if (live) {
            c.vx[s] = z.stage[2][s];
            c.vy[s] = z.stage[3][s];
            c.q[s] = z.stage[4][s];
            c.m[s] = z.stage[5][s];
            c.invm[s] = __drcp_rn(z.stage[5][s]);
            c.orig[s] = z.orig_stage[s];
            write_stage_position(c, 0, s, z.stage[0][s], z.stage[1][s]);  // set 0 is the state: x, y
            const float4 A = c.pa[0][s];
            xh = A.x;
            yh = A.y;
        } else if (store) {
            write_padding(c, s);
            c.q[s] = 0.0;
            c.m[s] = 1.0;
        }
        store_group_box(c.gbox[0] + (s >> 5), live, xh, yh, store);
    } else if (mid_ready) {
        return;
    }
    if (mid) write_midpoint_group(c, s, live, c.gbox[1] + (s >> 5), store, dt);
}

// An upload in the caller's order (staging arrays 0..3: x, y, vx, vy) put
// straight into the cloud's current internal order, with position set 0 and
// the boxes of its 32-particle groups: charges, masses and the order itself
// stay where they are (the next re-sort starts from them).  An upload that
// changes the state leaves its number: a program that downloads and uploads
// the same state between steps keeps the order (and the bits) of one that
// only steps.
static __global__ void upload_internal_order(CloudDev c, SortScratch z, int upload) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= c.n_pad) return;  // whole warps: n_pad is a multiple of 64
    float xh = 0.0f, yh = 0.0f;
    if (s < c.n) {
        const int o = c.orig[s];
        const double x = z.stage[0][o], y = z.stage[1][o], vx = z.stage[2][o], vy = z.stage[3][o];
        if (!(x == c.x[s] && y == c.y[s] && vx == c.vx[s] && vy == c.vy[s])) *z.changed = upload;
        c.vx[s] = vx;
        c.vy[s] = vy;
        write_stage_position(c, 0, s, x, y);  // set 0 is the state: x, y
        const float4 A = c.pa[0][s];
        xh = A.x;
        yh = A.y;
    }
    store_group_box(c.gbox[0] + (s >> 5), s < c.n, xh, yh, true);
}

static __global__ void set_identity(int *orig, int n) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < n) orig[s] = s;
}

// out[orig[s]] = in[s] for up to four arrays (internal -> caller order).
static __global__ void scatter_to_caller(const int *__restrict__ orig, int n, const double *a0,
                                         const double *a1, const double *a2, const double *a3,
                                         double *o0, double *o1, double *o2, double *o3) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const int o = orig[s];
    if (a0) o0[o] = a0[s];
    if (a1) o1[o] = a1[s];
    if (a2) o2[o] = a2[s];
    if (a3) o3[o] = a3[s];
}

// Four arrays of n doubles copied element for element (coalesced on both
// sides): caller buffers in page-locked host memory read or written by the
// device itself over the host link, in place of four DMA copies.  err_src /
// err_dst (optional): the device error word copied along with them.
static __global__ void copy4(int n, const double *__restrict__ i0, const double *__restrict__ i1,
                             const double *__restrict__ i2, const double *__restrict__ i3, double *o0,
                             double *o1, double *o2, double *o3, const int *err_src, int *err_dst) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (err_dst && s == 0) *err_dst = *err_src;
    if (s >= n) return;
    o0[s] = i0[s];
    o1[s] = i1[s];
    o2[s] = i2[s];
    o3[s] = i3[s];
}

// out[s] = in[orig[s]] for up to two arrays (caller -> internal order).
static __global__ void gather_from_caller(const int *__restrict__ orig, int n, const double *i0,
                                          const double *i1, double *o0, double *o1) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const int o = orig[s];
    if (i0) o0[s] = i0[o];
    if (i1) o1[s] = i1[o];
}

}  // namespace dm
