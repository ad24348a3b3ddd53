// dm_misc.cuh -- O(N) and reduction kernels around the pair kernels:
// stage-position initialisation, the adaptive-dt distance test, FP64
// diagnostics and the peak-throughput probe.
#pragma once

#include "dm_fp64.cuh"

namespace dm {

// Writes position set 0 (two-float copies and filter bounds) and 1/m from the
// state, and the padding particles of every set.
static __global__ void init_positions(CloudDev c) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n_pad) return;
    if (i < c.n) {
        write_stage_position(c, 0, i, c.x[i], c.y[i]);
        c.invm[i] = __drcp_rn(c.m[i]);
    } else {
        write_padding(c, i);
        c.q[i] = 0.0;
        c.m[i] = 1.0;
    }
}

// Position set 1 (x2 = x + dt v/2) and its group boxes from the state, when
// the step before did not leave them for this dt (one warp per group).
static __global__ void prepare_midpoint(CloudDev c, double dt, const double *dt_dev) {
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if ((i & ~31) >= c.n) return;  // whole warp
    float xh = 0.0f, yh = 0.0f;
    if (i < c.n) {
        write_midpoint(c, i, c.x[i], c.y[i], c.vx[i], c.vy[i], dt_dev ? *dt_dev : dt);
        const float4 A = c.pa[1][i];
        xh = A.x;
        yh = A.y;
    }
    store_group_box(c.gbox[1] + (i >> 5), i < c.n, xh, yh, true);
}

// After an RK2 step under the caller's stream capture: its results, left in
// sets 2 and 3 because other blocks were still reading sets 0 and 1, become sets
// 0 (the state) and 1.  (Outside a capture the sets' pointers change places;
// this copy was 3.5 us of a 35 us step of 4095 particles.)
static __global__ void adopt_sets(CloudDev c, int ngroups) {
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
#pragma unroll
    for (int b = 0; b < 2; b++) {
        if (i < c.n) {
            c.px[b][i] = c.px[b + 2][i];
            c.py[b][i] = c.py[b + 2][i];
            c.pa[b][i] = c.pa[b + 2][i];
            c.pb[b][i] = c.pb[b + 2][i];
        }
        if (i < ngroups) c.gbox[b][i] = c.gbox[b + 2][i];
    }
}

// The step counter and force time of slot `from` to slot `to`.
static __global__ void copy_slot(CloudDev c, int from, int to) {
    pdl_wait();
    c.step_ctr[to] = c.step_ctr[from];
    c.time[to] = c.time[from];
}

// Boxes of every 32 consecutive groups of sets b and b + 1 (large clouds): one
// warp per super group and set.
static __global__ void super_bounds(CloudDev c, int b, int ngroups) {
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const int nsuper = (ngroups + 31) >> 5;
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (w >= 2 * nsuper) return;  // whole warp
    const int e = w / nsuper, s = w % nsuper, g = 32 * s + lane;
    float4 v = (g < ngroups) ? c.gbox[b + e][g] : make_float4(INFINITY, INFINITY, -INFINITY, -INFINITY);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        v.x = fminf(v.x, __shfl_xor_sync(0xffffffffu, v.x, o));
        v.y = fminf(v.y, __shfl_xor_sync(0xffffffffu, v.y, o));
        v.z = fmaxf(v.z, __shfl_xor_sync(0xffffffffu, v.z, o));
        v.w = fmaxf(v.w, __shfl_xor_sync(0xffffffffu, v.w, o));
    }
    if (lane == 0) c.gsuper[b + e][s] = v;
}

// Force time slots = t (see stage_time()).
static __global__ void set_time_slots(double *time, double t) {
    time[0] = t;
    time[1] = t;
}

// For the autotuner: the positions squeezed about (cx, cy) by lam, written
// as position set 1, so kernels can be timed on a denser copy of the cloud
// without touching its state.
static __global__ void tune_compress(CloudDev c, double cx, double cy, double lam) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < c.n) write_stage_position(c, 1, i, cx + lam * (c.x[i] - cx), cy + lam * (c.y[i] - cy));
}

// Bounding box of each 32-particle group's FP32 positions (hi parts) in
// position set b, for the culling pair kernels: one warp per group; padding
// particles are left out, so an all-padding group gets an empty box.
static __global__ void group_bounds(CloudDev c, int b) {
    pdl_wait();
    const int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const int i = 32 * g + lane;
    if (32 * g >= c.n_pad) return;  // whole warp
    const float4 A = (i < c.n) ? c.pa[b][i] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    store_group_box(c.gbox[b] + g, i < c.n, A.x, A.y, true);
}

// ---------------------------------------------------------------------------
// Adaptive dt (Integrator::modifyTimeStep, Integrator.cpp:68-134).
// Pairs checked: all 6 pairs inside each 4-block; between 4-blocks o < p,
// element k of o with element (k - d) mod 4 of p for d = 0, 1, 2.
// Separations are computed from (float)x exactly as the SSE code does
// (sub, mul, mul, add, sqrt in FP32, no fused multiply-add).
// ---------------------------------------------------------------------------
__device__ __forceinline__ float sep2_f32(float ax, float ay, float bx, float by) {
    const float sx = __fsub_rn(ax, bx), sy = __fsub_rn(ay, by);
    return __fadd_rn(__fmul_rn(sx, sx), __fmul_rn(sy, sy));
}

// The separations are FP32, so the positions are rounded once per particle (in
// the caller's order, which defines the pairs), not once per pair.
static __global__ void adaptive_positions(CloudDev c, float2 *__restrict__ p, unsigned int *min_done) {
    pdl_wait();
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s == 0) {
        min_done[0] = 0x7f7f7f7fu;
        min_done[1] = 0u;
    }
    if (s < c.n) p[c.orig[s]] = make_float2(__double2float_rn(c.x[s]), __double2float_rn(c.y[s]));
}

// tryToReduceTimeStep (Integrator.cpp:144-155) applied to the minimum:
// while dmin <= dist: dist /= 10.0f, dt /= 10.0.  A zero separation (where
// the reference never terminates) sets error bit 2 and leaves dt unchanged.
struct AdaptiveResult {
    double dt;
    float dmin;
    int err;
};
__device__ __forceinline__ AdaptiveResult adaptive_dt(float min_r2, double init_dt, int *err) {
    AdaptiveResult R{init_dt, __fsqrt_rn(min_r2), 0};
    float dist = 1.0e-4f;
    if (R.dmin > 0.0f) {
        for (int it = 0; it < 200 && R.dmin <= dist; it++) {
            dist = __fdiv_rn(dist, 10.0f);
            R.dt = __ddiv_rn(R.dt, 10.0);
        }
        R.err = atomicOr(err, 0);
    } else {
        R.err = atomicOr(err, 2) | 2;
    }
    return R;
}

// The minimum over the checked pairs of the nb 4-blocks, then the time step.
// Tiles of 32 x 32 4-blocks of the upper triangle, grid-strided: a lane keeps
// one outer block, a warp goes through the tile's inner blocks.  The minimum
// r^2 (a non-negative float, so its bit pattern orders like an unsigned int)
// is combined with atomicMin, which is order-independent; the block that is
// last (min_done[1] counts them) forms the result, on the device (dt_out) and
// in page-locked host memory.  Bound by launch and memory latency:
// 2048 particles 4.8 us, 6 us with the rounding launch (converting both
// positions of every pair, and the copy, reset and result launches around it,
// took 15 us).
constexpr int kAdaptTile = 32;
static __global__ void __launch_bounds__(256) checked_min_dist2(const float2 *__restrict__ pos, int nb, double init_dt,
                                                                unsigned int *min_done, double *dt_out, int *err,
                                                                AdaptiveResult *host) {
    pdl_wait();
    __shared__ float4 tile[kAdaptTile][2];  // an inner 4-block: its positions in pairs
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nt = (nb + kAdaptTile - 1) / kAdaptTile;
    const long long total = (long long)nt * (nt + 1) / 2;
    const float4 *__restrict__ p4 = reinterpret_cast<const float4 *>(pos);
    float best = INFINITY;
    for (long long t = blockIdx.x; t < total; t += gridDim.x) {
        // row r of the triangle's transpose holds tiles (q, r), q = 0 .. r
        long long r = (long long)(0.5f * (sqrtf(8.0f * (float)t + 1.0f) - 1.0f));
        while (r * (r + 1) / 2 > t) r--;
        while ((r + 1) * (r + 2) / 2 <= t) r++;
        const int o = (int)(t - r * (r + 1) / 2) * kAdaptTile + lane;
        const int p0 = (int)r * kAdaptTile;
        __syncthreads();
        if (threadIdx.x < 2 * kAdaptTile) {
            const int e = 2 * p0 + (int)threadIdx.x;
            tile[threadIdx.x >> 1][threadIdx.x & 1] = (e < 2 * nb) ? p4[e] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
        __syncthreads();
        const bool in = o < nb;
        const float4 a = p4[in ? 2 * o : 0], b = p4[in ? 2 * o + 1 : 1];
        const float ox[4] = {a.x, a.z, b.x, b.z}, oy[4] = {a.y, a.w, b.y, b.w};
        for (int k = warp; k < kAdaptTile && p0 + k < nb; k += 8) {
            const int p = p0 + k;
            if (!in || p < o) continue;
            if (p == o) {
                const int ia[6] = {0, 2, 0, 1, 1, 0}, ib[6] = {1, 3, 3, 2, 3, 2};
#pragma unroll
                for (int e = 0; e < 6; e++) best = fminf(best, sep2_f32(ox[ia[e]], oy[ia[e]], ox[ib[e]], oy[ib[e]]));
            } else {
                const float4 u = tile[k][0], v = tile[k][1];
                const float ix[4] = {u.x, u.z, v.x, v.z}, iy[4] = {u.y, u.w, v.y, v.w};
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int d = 0; d < 3; d++) {
                        const int m = (i - d + 4) & 3;
                        best = fminf(best, sep2_f32(ox[i], oy[i], ix[m], iy[m]));
                    }
            }
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) best = fminf(best, __shfl_xor_sync(0xffffffffu, best, off));
    if (lane == 0) {
        atomicMin(min_done, __float_as_uint(best));
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(min_done + 1, 1u) == gridDim.x - 1) {
        const AdaptiveResult R = adaptive_dt(__uint_as_float(atomicMin(min_done, 0xffffffffu)), init_dt, err);
        *dt_out = R.dt;
        *host = R;
    }
}

// ---------------------------------------------------------------------------
// FP64 diagnostics: per-block partial sums of kinetic energy, Yukawa
// potential (kappa*r < 10, counted once per unordered pair), confinement
// potential and momentum, written to partial[blockIdx.x*5 + ...] and summed
// in block order by diagnostics_finish.
//
// The pairs (I, J >= I) of 256-particle tiles are dealt to a grid of at most
// kDiagBlocks blocks (so the order of every sum depends on n alone).  A warp
// filters 32 particles of tile I against tile J in FP32, from positions
// rounded to FP32 with a bound that covers the rounding, and evaluates the
// hits in FP64 32 at a time (dm_fp64.cuh).  Bound by the filter's issue slots
// (~7 per 32 pairs) on sparse clouds, by the FP64 pipe on dense ones.
// ---------------------------------------------------------------------------
constexpr int kDiagTile = 256;
constexpr int kDiagBlocks = 608;

struct DiagSmem {
    double x[2][kDiagTile], y[2][kDiagTile], q[2][kDiagTile];  // tiles I and J
    float2 f[kDiagTile];                                        // tile J in FP32
    double tab[kExp2Size];
    uint32_t mask[kDiagTile / 32][kDiagTile / 32][32];
    uint16_t code[kDiagTile / 32][kHitSumPerLane * 32];
    double red[kDiagTile / 32][5];
    unsigned int amax;
};

static __global__ void __launch_bounds__(kDiagTile) diagnostics_partial(const CloudDev c, const ForceParams f,
                                                                        const Yukawa64 K, double rc, double coulomb,
                                                                        double *partial) {
    __shared__ DiagSmem sm;
    constexpr int NG = kDiagTile / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int k = tid; k < kExp2Size; k += kDiagTile) sm.tab[k] = g_exp2_table.v[k];
    double v[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    double pe = 0.0;
    const int nb = (c.n + kDiagTile - 1) / kDiagTile;
    const long long total = (long long)nb * (nb + 1) / 2;
    int have = -1, I = 0;
    long long row = 0;  // first pair index of row I
    for (long long p = blockIdx.x; p < total; p += gridDim.x) {
        while (p >= row + nb - I) {
            row += nb - I;
            I++;
        }
        const int J = I + (int)(p - row);
        const int i = I * kDiagTile + tid, j = J * kDiagTile + tid;
        __syncthreads();  // the previous pair's tiles are done with
        if (I != have) {
            have = I;
            sm.x[0][tid] = (i < c.n) ? c.x[i] : 0.0;
            sm.y[0][tid] = (i < c.n) ? c.y[i] : 0.0;
            sm.q[0][tid] = (i < c.n) ? c.q[i] : 0.0;
        }
        if (I == J && i < c.n) {  // the tile's one-particle terms
            const double x = c.x[i], y = c.y[i], vx = c.vx[i], vy = c.vy[i], q = c.q[i], m = c.m[i];
            v[0] += 0.5 * m * (vx * vx + vy * vy);
            v[3] += m * vx;
            v[4] += m * vy;
            if (f.flags & kConfinement) v[2] += -0.5 * q * f.confine * (x * x + y * y);
            if (f.flags & kRectConfinement) v[2] += -0.5 * q * (f.confine_x * x * x + f.confine_y * y * y);
        }
        if (!(f.flags & kShieldedCoulomb)) continue;
        float2 fj = make_float2(0.0f, 0.0f);
        if (j < c.n) {
            const double x = c.x[j], y = c.y[j];
            sm.x[1][tid] = x;
            sm.y[1][tid] = y;
            sm.q[1][tid] = c.q[j];
            fj = make_float2(__double2float_rn(x), __double2float_rn(y));
        }
        sm.f[tid] = fj;
        if (tid == 0) sm.amax = 0u;
        __syncthreads();
        // largest |coordinate| of the tile (NaN has the largest bits: every
        // pair of the tile is then a candidate)
        const uint32_t am = __reduce_max_sync(
            0xffffffffu, max(__float_as_uint(fabsf(fj.x)), __float_as_uint(fabsf(fj.y))));
        if (lane == 0) atomicMax(&sm.amax, am);
        __syncthreads();
        const float xf = __double2float_rn(sm.x[0][tid]), yf = __double2float_rn(sm.y[0][tid]);
        const float bound =
            candidate_bound(rc, fmaxf(fabsf(xf), fabsf(yf)), __uint_as_float(sm.amax));
        const int left = c.n - J * kDiagTile;
        for (int k = 0; k < NG; k++) {
            uint32_t m = 0u;
            if (I < J || k >= warp) {  // tile against itself: groups k >= the warp's
#pragma unroll 8
                for (int u = 31; u >= 0; u--) {
                    const float2 A = sm.f[32 * k + u];
                    const float dx = xf - A.x, dy = yf - A.y;
                    m = 2u * m + (fmaf(dx, dx, dy * dy) >= bound ? 0u : 1u);
                }
                if (I == J && k == warp) m &= ~((2u << lane) - 1u);  // j > i
                if (left < 32 * k + 32) m &= (left > 32 * k) ? (1u << (left - 32 * k)) - 1u : 0u;
                if (i >= c.n) m = 0u;
            }
            sm.mask[warp][k][lane] = m;
        }
        __syncwarp();
        hit_sum(sm.mask[warp], NG, sm.code[warp], [&](int il, int jl) {
            const int a = 32 * warp + il;
            const double dx = __dsub_rn(sm.x[0][a], sm.x[1][jl]), dy = __dsub_rn(sm.y[0][a], sm.y[1][jl]);
            const double r2 = fma(dx, dx, __dmul_rn(dy, dy));
            const Yukawa64At A = yukawa64_odd(r2) ? yukawa64_general(r2, K.kappa) : yukawa64(r2, K, sm.tab);
            const double e = __dmul_rn(__dmul_rn(sm.q[0][a], sm.q[1][jl]), __dmul_rn(A.ex, A.y));
            if (in_cutoff64(dx, dy, r2, K)) pe = __dadd_rn(pe, e);
        });
    }
    v[1] = __dmul_rn(coulomb, pe);
#pragma unroll
    for (int e = 0; e < 5; e++) {
        double t = v[e];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) sm.red[warp][e] = t;
    }
    __syncthreads();
    if (tid < 5) {
        double t = 0.0;
        for (int w = 0; w < NG; w++) t += sm.red[w][tid];
        partial[blockIdx.x * 5 + tid] = t;
    }
}

// Sums the per-block partials into out[0..4]: warp e takes quantity e, lanes
// strided over the blocks, then a butterfly.
static __global__ void __launch_bounds__(160) diagnostics_finish(const double *partial, int nblocks, double *out) {
    const int lane = threadIdx.x & 31, e = threadIdx.x >> 5;
    double t = 0.0;
    for (int b = lane; b < nblocks; b += 32) t += partial[b * 5 + e];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) out[e] = t;
}

inline int diagnostics_blocks(int n) {
    const long long nb = (n + kDiagTile - 1) / kDiagTile;
    const long long pairs = nb * (nb + 1) / 2;
    return (int)(pairs < kDiagBlocks ? pairs : kDiagBlocks);
}

// ---------------------------------------------------------------------------
// Peak probe: 16 independent FMA chains per thread.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void fma_probe(T *out, int iters, T a, T b) {
    T acc[16];
#pragma unroll
    for (int k = 0; k < 16; k++) acc[k] = (T)(threadIdx.x + k);
    for (int it = 0; it < iters; it++) {
#pragma unroll
        for (int k = 0; k < 16; k++) acc[k] = acc[k] * a + b;
    }
    T s = 0;
#pragma unroll
    for (int k = 0; k < 16; k++) s += acc[k];
    if (s == (T)-1.2345) out[0] = s;  // keeps the loop alive
}

}  // namespace dm
