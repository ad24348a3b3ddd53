// dm_batch.cuh -- many independent clouds of uneven size in one launch.
//
// The clouds are concatenated (caller order: cloud 0's particles, then cloud
// 1's, ...) into one set of device arrays with no per-cloud padding; each
// cloud keeps its own force parameters (kappa, charge, confinement, ...).
// The pair forces of a pass (two RK stages, see dm_device.cuh) are ONE launch:
// a work item is a (cloud, i-tile, position set), taken by one block that runs
// the same FP32C sweep as the single-cloud kernel over that cloud's j and
// leaves the tile's sums in global memory; batch_finish then runs the epilogue
// of every 32-particle group.  (In one launch, the blocks' epilogues -- chains
// of FP64 operations on two of a block's warps -- kept the registers and
// shared memory of the sweep occupied while they ran.)  Items are ordered by
// cost (largest clouds first) and blocks start in that order as SMs free up, a
// longest-processing-time schedule; an item is computed entirely by one
// block, so the result does not depend on where it runs (deterministic, no
// atomics on forces).
#pragma once

#include "dm_pair.cuh"
#include "dm_sort.cuh"

namespace dm {

struct BatchCloud {
    int off;        // first particle in the concatenated arrays
    int n;
    int goff;       // first of the cloud's 32-particle groups in the batch's group boxes
    ForceParams f;
    double rc2;
    float rc2_lo, rc2_hi, rc2_up, kappa_f;
    float nkl2e;    // -kappa*log2(e)
};

// A work item: a tile of a cloud, the cloud's first particle and size.
struct BatchItem {
    int cloud, tile, off, n;
};

// ... of a batch's cloud by value, in shared memory (see StageView).
struct SweepView {
    const float4 *pa_, *pb_;
    const double *px_, *py_;
    const float4 *gbox_;
    unsigned long long *eval_pairs_;
    double kappa_;
    int n_;
    float rc2_lo_, rc2_hi_, kappa_f_, nkl2e_;
    int direct_min_;
    float near_direct_f2_;
    __device__ __forceinline__ int n() const { return n_; }
    __device__ __forceinline__ const float4 *pa() const { return pa_; }
    __device__ __forceinline__ const float4 *pb() const { return pb_; }
    __device__ __forceinline__ const double *px() const { return px_; }
    __device__ __forceinline__ const double *py() const { return py_; }
    __device__ __forceinline__ const float4 *gbox() const { return gbox_; }
    __device__ __forceinline__ const float4 *gsuper() const { return nullptr; }
    __device__ __forceinline__ unsigned long long *eval_pairs() const { return eval_pairs_; }
    __device__ __forceinline__ double kappa() const { return kappa_; }
    __device__ __forceinline__ float rc2_lo() const { return rc2_lo_; }
    __device__ __forceinline__ float rc2_hi() const { return rc2_hi_; }
    __device__ __forceinline__ float kappa_f() const { return kappa_f_; }
    __device__ __forceinline__ float nkl2e() const { return nkl2e_; }
    __device__ __forceinline__ int direct_min() const { return direct_min_; }
    __device__ __forceinline__ float near_direct_f2() const { return near_direct_f2_; }
};

// Only what the sweep reads is fetched of a cloud's record, by one thread, and
// the item itself holds the cloud's place (256 clouds: 221 us a launch; with a
// copy of all the launch's parameters per block 242 us).
template <int NW, int ILP, int TC, bool CULL = false>
__global__ void __launch_bounds__(NW * 32, fp32c_min_blocks<NW, ILP>())
    batch_stage_fp32c(const StageParams P, const BatchCloud *__restrict__ desc, const BatchItem *__restrict__ items) {
    constexpr int TILE = 32 * ILP;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ SweepView V;
    const float4 *s_red = reinterpret_cast<const float4 *>(smem_raw) + Fp32cSmem<NW, ILP, TC>::red_offset;
    pdl_wait();
    const int set = blockIdx.x % P.nsets;
    const BatchItem w = items[blockIdx.x / P.nsets];
    if (threadIdx.x == 0) {
        const BatchCloud &d = desc[w.cloud];
        const CloudDev &c = P.c;
        const int b = P.buf[set];
        V = {c.pa[b] + w.off, c.pb[b] + w.off, c.px[b] + w.off, c.py[b] + w.off, c.gbox[b] + d.goff,
             c.eval_pairs,    d.f.shielding,   w.n,             d.rc2_lo,        d.rc2_hi,           d.kappa_f,
             d.nkl2e,         P.direct_min,    P.near_direct_f2};
    }
    __syncthreads();
    fp32c_sweep<NW, ILP, TC, CULL>(V, w.tile, 0, 1, threadIdx.x, [] { __syncthreads(); }, smem_raw);
    const int first = w.off + w.tile * TILE, n = min(TILE, w.n - w.tile * TILE);
    for (int e = threadIdx.x; e < n; e += NW * 32) {
        const float4 v = s_red[e];
        P.partial[(size_t)(2 * set) * P.c.n_pad + first + e] = make_float2(v.x, v.z);
        P.partial[(size_t)(2 * set + 1) * P.c.n_pad + first + e] = make_float2(v.y, v.w);
    }
}

// The pass's epilogue for every 32-particle group of every cloud (group w is
// of cloud gseg[w]): one block of two warps each.
static __global__ void __launch_bounds__(64) batch_finish(const StageParams P, const BatchCloud *__restrict__ desc,
                                                          const int *__restrict__ gseg) {
    __shared__ EpilogueShared S;
    pdl_wait();
    const int lane = threadIdx.x & 31, ax = threadIdx.x >> 5;
    const BatchCloud &d = desc[gseg[blockIdx.x]];
    const int li = 32 * ((int)blockIdx.x - d.goff) + lane, i = d.off + li;
    const bool live = li < d.n;
    double f[2] = {0.0, 0.0};
    if (live) {
        epilogue_prefetch(P, i, ax);
        for (int e = 0; e < P.nsets; e++) f[e] = finish_rank_sum(P, i, e, ax);
    }
    pass_epilogue(P, EpilogueCloud{d.f, d.rc2_up, live, (int)blockIdx.x}, i, ax, kBarEpilogue, f[0], f[1], S);
    pass_step_advance(P);
}

// Box of every cloud's 32-particle groups in position set b (one warp per
// group; gseg[w] is group w's cloud; a cloud's last group may be partial).
static __global__ void batch_group_bounds(CloudDev c, const BatchCloud *__restrict__ desc,
                                          const int *__restrict__ gseg, int ngroups, int b) {
    pdl_wait();
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (w >= ngroups) return;  // whole warp
    const BatchCloud &d = desc[gseg[w]];
    const int li = 32 * (w - d.goff) + lane;
    const float4 A = (li < d.n) ? c.pa[b][d.off + li] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    store_group_box(c.gbox[b] + w, li < d.n, A.x, A.y, true);
}

// Position set 1 (the step's midpoint) of every cloud, when the step before
// did not leave it for this dt.
static __global__ void batch_midpoint(CloudDev c, const BatchCloud *__restrict__ desc, const int *__restrict__ seg,
                                      double dt) {
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n) return;
    CloudDev v = c;
    v.rc2_up = desc[seg[i]].rc2_up;
    write_midpoint(v, i, c.x[i], c.y[i], c.vx[i], c.vy[i], dt);
}

// --- per-cloud Morton order ------------------------------------------------

// One block per cloud: the cloud's key box (the bounding box clipped to
// mean +- 4 sigma per axis) and bounding box, box[8 * cloud ...] as in
// moments_to_box.  Deterministic (fixed partition and order).
static __global__ void __launch_bounds__(256) batch_boxes(const double *__restrict__ x,
                                                          const double *__restrict__ y,
                                                          const BatchCloud *__restrict__ desc, double *box) {
    const BatchCloud &d = desc[blockIdx.x];
    const double ox = finite_or_zero(x[d.off]), oy = finite_or_zero(y[d.off]);
    const Moments m = block_moments(x, y, d.off, d.off + d.n, blockDim.x, ox, oy);
    if (threadIdx.x == 0) moments_to_box(m, ox, oy, box + 8 * blockIdx.x);
}

// key = cloud index (high bits) | the top `mbits` bits of the 24-bit Morton
// code within the cloud's box, so a stable sort keeps every cloud in its own
// contiguous range.
static __global__ void batch_keys(const double *__restrict__ x, const double *__restrict__ y, int n,
                                  const int *__restrict__ seg, const double *__restrict__ box,
                                  int mbits, uint32_t *keys, int *vals) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int sg = seg[i];
    const double *bb = box + 8 * sg;
    const double x0 = bb[0], y0 = bb[1], ext = bb[2];
    const double scale = (ext > 0.0 && isfinite(ext)) ? 4095.0 / ext : 0.0;
    const double fx = (x[i] - x0) * scale, fy = (y[i] - y0) * scale;
    const uint32_t qx = (fx > 0.0) ? (uint32_t)fmin(fx, 4095.0) : 0u;
    const uint32_t qy = (fy > 0.0) ? (uint32_t)fmin(fy, 4095.0) : 0u;
    const uint32_t morton = spread_bits12(qx) | (spread_bits12(qy) << 1);
    keys[i] = ((uint32_t)sg << mbits) | (morton >> (24 - mbits));
    vals[i] = i;
}

// ---------------------------------------------------------------------------
// Per-cloud sort for batches whose clouds all hold at most kBatchSortMax
// particles: block b sorts cloud b on its own -- key box, 24-bit Morton keys,
// three stable 8-bit LSD passes in shared memory -- gathers the cloud's state
// in the new order into registers and, after a block barrier (the block holds
// the whole cloud), rewrites the cloud's arrays in place with position sets 0
// and 1 and their group boxes.  One launch replaces the batch-wide path
// (per-cloud boxes, keys with the cloud index in the high bits, four radix
// passes over every particle of every cloud, gather: a dozen dependent
// launches).  As in sort_cluster the key box and keys are FP32 functions of
// the positions' hi parts (set 0), lanes with equal digits are found by
// match_digit8, and the element order (warp, round, lane) makes every pass
// stable.
// ---------------------------------------------------------------------------
constexpr int kBatchSortMax = 4096;
constexpr int kBatchSortThreads = 1024;
constexpr int kBatchSortWarps = kBatchSortThreads / 32;
constexpr int kBatchSortRounds = kBatchSortMax / kBatchSortThreads;  // 4 per thread

struct BatchSortSmem {
    uint32_t keys[2][kBatchSortMax];
    uint16_t slot[2][kBatchSortMax];
    uint32_t wcnt[kBatchSortWarps][kSortBuckets];  // per-warp digit counts, then offsets
    uint32_t dbase[kSortBuckets];
    uint32_t part[kSortBuckets / 32];
    float wmom[kBatchSortWarps][kMomentFields];
    float box[3];
};
constexpr size_t kBatchSortSmem = sizeof(BatchSortSmem);

// box_out[8 * cloud]: key box x0, y0, extent, -, bounding box min x, min y, max
// x, max y (as batch_boxes writes them; the batch autotuner reads it).  Without `force` a cloud in good order (see
// kOrderKeep) is left as it is; if `mid` and not `mid_ready` its set 1 is
// written.  order[cloud]: its last sort; slot: of the step counter.
static __global__ void __launch_bounds__(kBatchSortThreads, 1)
    batch_sort_clouds(CloudDev c, const BatchCloud *__restrict__ desc, double *box_out, double dt, bool mid,
                      bool mid_ready, bool force, int slot, OrderRecord *order) {
    pdl_wait();
    extern __shared__ __align__(128) unsigned char smem_raw[];
    BatchSortSmem &S = *reinterpret_cast<BatchSortSmem *>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const OrderRecord was = order[blockIdx.x];
    const unsigned long long step = c.step_ctr[slot];
    const BatchCloud d = desc[blockIdx.x];
    const int off = d.off, n = d.n;
    const float4 *__restrict__ pa0 = c.pa[0] + off;
    const int groups = (n + 31) / 32;

    if (!force && order_is_recent(step, was.step)) {
        const OrderRecord now = block_order_record<1>(c.gbox[0] + d.goff, pa0, groups, S.wmom);
        if (order_is_good(now, was, groups, sqrtf(d.rc2_up))) {
            if (mid && !mid_ready) {
                CloudDev v = c;
                v.rc2_up = d.rc2_up;
                for (int k = 0; k < kBatchSortRounds; k++) {
                    const int li = k * kBatchSortThreads + tid;
                    write_midpoint_group(v, off + li, li < n, c.gbox[1] + d.goff + (li >> 5), (li & ~31) < n, dt);
                }
            }
            return;
        }
    }

    float4 pos[kBatchSortRounds];
#pragma unroll
    for (int k = 0; k < kBatchSortRounds; k++) {
        const int e = k * kBatchSortThreads + tid;
        pos[k] = (e < n) ? pa0[e] : make_float4(NAN, NAN, 0.0f, 0.0f);
    }
    const float4 p0 = pa0[0];
    const float ox = isfinite(p0.x) ? p0.x : 0.0f, oy = isfinite(p0.y) ? p0.y : 0.0f;
    {
        float v[kMomentFields] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, INFINITY, INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int k = 0; k < kBatchSortRounds; k++) moments_f32_add(v, pos[k], ox, oy);
        moments_f32_block<kBatchSortWarps>(v, S.wmom);
        if (tid == 0) {
            key_box_f32(v, ox, oy, S.box);
            double *bo = box_out + 8 * blockIdx.x;
            bo[0] = S.box[0];
            bo[1] = S.box[1];
            bo[2] = S.box[2];
            for (int k = 0; k < 4; k++) bo[4 + k] = (v[0] > 0.0f) ? (double)v[5 + k] : 0.0;
        }
        __syncthreads();
    }
#pragma unroll
    for (int k = 0; k < kBatchSortRounds; k++) {
        const int li = k * kBatchSortThreads + tid;
        S.keys[0][li] = (li < n) ? morton_key_f32(pos[k].x, pos[k].y, S.box) : 0u;
        S.slot[0][li] = (uint16_t)li;
    }
    __syncthreads();

    const uint32_t lower = (1u << lane) - 1u;
    int cur = 0;
    for (int shift = 0; shift < kSortBits; shift += kSortDigitBits) {
        for (int dg = lane; dg < kSortBuckets; dg += 32) S.wcnt[warp][dg] = 0u;
        __syncwarp();
        uint32_t dk[kBatchSortRounds], rk[kBatchSortRounds];
#pragma unroll
        for (int k = 0; k < kBatchSortRounds; k++) {
            const int li = warp * (32 * kBatchSortRounds) + k * 32 + lane;
            const bool valid = li < n;
            const uint32_t dg = (S.keys[cur][li] >> shift) & (kSortBuckets - 1);
            const uint32_t peers = match_digit8(dg, valid);
            rk[k] = S.wcnt[warp][dg] + __popc(peers & lower);
            dk[k] = valid ? dg : kSortBuckets;
            __syncwarp();
            if (valid && (peers & lower) == 0u) S.wcnt[warp][dg] += __popc(peers);
            __syncwarp();
        }
        __syncthreads();
        uint32_t tot = 0u, inc = 0u;
        if (tid < kSortBuckets) {  // per digit: offsets of the warps, block total, scan over digits
            for (int w = 0; w < kBatchSortWarps; w++) {
                const uint32_t v = S.wcnt[w][tid];
                S.wcnt[w][tid] = tot;
                tot += v;
            }
            inc = tot;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += v;
            }
            if (lane == 31) S.part[warp] = inc;
        }
        __syncthreads();
        if (tid < kSortBuckets) {
            uint32_t wb = 0u;
            for (int w = 0; w < warp; w++) wb += S.part[w];
            S.dbase[tid] = wb + inc - tot;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kBatchSortRounds; k++) {
            if (dk[k] < (uint32_t)kSortBuckets) {
                const int li = warp * (32 * kBatchSortRounds) + k * 32 + lane;
                const uint32_t p = S.dbase[dk[k]] + S.wcnt[warp][dk[k]] + rk[k];
                if (p >= (uint32_t)n) {  // cannot happen for a consistent count; never store out of range
                    atomicOr(c.err, kErrSortPermutation);
                    continue;
                }
                S.keys[cur ^ 1][p] = S.keys[cur][li];
                S.slot[cur ^ 1][p] = S.slot[cur][li];
            }
        }
        __syncthreads();
        cur ^= 1;
    }

    // gather the cloud's state in the new order (all loads before the stores)
    int src[kBatchSortRounds];
#pragma unroll
    for (int k = 0; k < kBatchSortRounds; k++) {
        const int li = k * kBatchSortThreads + tid;
        int o = (li < n) ? (int)S.slot[cur][li] : 0;
        if (li < n && o >= n) {
            atomicOr(c.err, kErrSortPermutation);
            o = li;
        }
        src[k] = off + o;
    }
    const double *in[6] = {c.x, c.y, c.vx, c.vy, c.q, c.m};
    double val[6][kBatchSortRounds];
    int ov[kBatchSortRounds];
#pragma unroll
    for (int k = 0; k < kBatchSortRounds; k++) {
        const bool ok = k * kBatchSortThreads + tid < n;
#pragma unroll
        for (int a = 0; a < 6; a++) val[a][k] = ok ? in[a][src[k]] : 0.0;
        ov[k] = ok ? c.orig[src[k]] : 0;
    }
    __syncthreads();  // every source is in registers: the cloud is rewritten in place
    CloudDev v = c;
    v.rc2_up = d.rc2_up;
#pragma unroll
    for (int k = 0; k < kBatchSortRounds; k++) {
        const int li = k * kBatchSortThreads + tid, s = off + li;  // a warp holds 32 consecutive slots
        float2 h[2] = {};
        if (li < n) {
            c.vx[s] = val[2][k];
            c.vy[s] = val[3][k];
            c.q[s] = val[4][k];
            c.m[s] = val[5][k];
            c.invm[s] = __drcp_rn(val[5][k]);
            c.orig[s] = ov[k];
            write_stage_position(v, 0, s, val[0][k], val[1][k]);  // set 0 is the state: x, y
            h[0] = make_float2(__double2float_rn(val[0][k]), __double2float_rn(val[1][k]));
            if (mid) {
                write_midpoint(v, s, val[0][k], val[1][k], val[2][k], val[3][k], dt);
                const float4 A = c.pa[1][s];
                h[1] = make_float2(A.x, A.y);
            }
        }
        store_group_box(c.gbox[0] + d.goff + (li >> 5), li < n, h[0].x, h[0].y, (li & ~31) < n);
        if (mid) store_group_box(c.gbox[1] + d.goff + (li >> 5), li < n, h[1].x, h[1].y, (li & ~31) < n);
    }
    __syncthreads();  // the boxes are written
    OrderRecord now = block_order_record<1>(c.gbox[0] + d.goff, c.pa[0] + off, groups, S.wmom);
    now.step = step;
    if (tid == 0) order[blockIdx.x] = now;
}

// For the batch autotuner: every cloud squeezed about its own box centre
// so that ~30% of its pairs are inside its cutoff (clouds already that dense
// are copied as they are), written as position set 1.
static __global__ void batch_tune_compress(CloudDev c, const BatchCloud *__restrict__ desc,
                                           const int *__restrict__ seg, const double *__restrict__ box) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n) return;
    const int sg = seg[i];
    const double *bb = box + 8 * sg;  // bounding box in bb[4..7]
    const double x0 = bb[4], y0 = bb[5], x1 = bb[6], y1 = bb[7];
    const double half = 0.5 * fmax(x1 - x0, y1 - y0);
    double lam = 1.8 * sqrt(desc[sg].rc2) / half;
    if (!(isfinite(lam) && lam > 0.0 && lam < 1.0)) lam = 1.0;
    const double cx = 0.5 * (x0 + x1), cy = 0.5 * (y0 + y1);
    CloudDev v = c;
    v.rc2_up = desc[sg].rc2_up;
    write_stage_position(v, 1, i, cx + lam * (c.x[i] - cx), cy + lam * (c.y[i] - cy));
}

// After permute_gather: the state in its new order, with position set 0 (each
// particle's own cloud's filter bound) and the padding.
static __global__ void batch_commit(CloudDev c, const BatchCloud *__restrict__ desc, const int *__restrict__ seg,
                                    SortScratch z) {
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < c.n) {
        c.vx[i] = z.stage[2][i];
        c.vy[i] = z.stage[3][i];
        c.q[i] = z.stage[4][i];
        c.m[i] = z.stage[5][i];
        c.invm[i] = __drcp_rn(z.stage[5][i]);
        c.orig[i] = z.orig_stage[i];
        CloudDev v = c;
        v.rc2_up = desc[seg[i]].rc2_up;
        write_stage_position(v, 0, i, z.stage[0][i], z.stage[1][i]);
    } else if (i < c.n_pad) {
        write_padding(c, i);
    }
}

// Position set 0 from the state, with each particle's own cloud's filter
// bound, 1/m, and the padding.
static __global__ void batch_init_positions(CloudDev c, const BatchCloud *__restrict__ desc,
                                            const int *__restrict__ seg) {
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < c.n) {
        CloudDev v = c;
        v.rc2_up = desc[seg[i]].rc2_up;
        write_stage_position(v, 0, i, c.x[i], c.y[i]);
        c.invm[i] = __drcp_rn(c.m[i]);
    } else if (i < c.n_pad) {
        write_padding(c, i);
    }
}

}  // namespace dm
