// dm_pair.cuh -- tiled all-pairs shielded-Coulomb (Yukawa) kernels with the
// RK4 stage epilogue fused in, for sm_103a.
//
// Replaces ShieldedCoulombForce::force1..4 (ShieldedCoulombForce.cpp:37-237)
// plus, in the epilogue, the per-particle forces, CacheOperator and the RK
// stage/combine loops (see dm_device.cuh).
//
// Work decomposition (owner computes, no atomics on forces), for each of the
// pass's position sets (dm_device.cuh):
//   * an i-tile of 32*ILP particles belongs to S CTAs (with the other set's S
//     CTAs a thread-block cluster, or plain blocks whose partial sums
//     stage_finish adds); lane l of every warp of those CTAs owns particles i
//     = tile*32*ILP + k*32 + l, k < ILP (the lane's i "slots"), in registers;
//   * rank r of the S sweeps every S-th chunk of 4 j (or, culling, every
//     S-th of the 32-particle j groups within reach of the tile), staging them
//     in shared memory; the CTA's warps deal the staged chunks round-robin;
//   * pairs of groups that may hold a pair within the cutoff are first
//     filtered with the expanded distance |p_j|^2 - 2 p_i.p_j against a per-i
//     bound (two j per packed FMA) -- the GPU form of the reference's early
//     exit for kappa*r >= 10 (ShieldedCoulombForce.cpp:178-180); groups
//     entirely within the cutoff skip the filter;
//   * the pair terms are evaluated two j at a time in packed f32x2
//     arithmetic (pair2_terms); the per-particle sums are compensated and the
//     pass's epilogue runs once per particle in FP64.
#pragma once

#include <cooperative_groups.h>

#include <type_traits>

#include "dm_device.cuh"
#include "dm_fp64.cuh"

namespace dm {
namespace cg = cooperative_groups;

// e^{-kappa r} on the SFU with kappa*log2(e) = k_hi + k_lo given as a float
// pair: t = k_hi r rounded to FP32 (absolute error up to ~1e-6 at kappa r =
// 10), and its residue t_lo (exact to ~2^-48) put back to first order,
// 2^{-(t + t_lo)} = 2^{-t} (1 - t_lo ln 2).  Relative error: the hardware
// ex2.approx (a few ulp) plus (t_lo ln 2)^2 / 2 < 1e-12, for the FP32 r given.
__device__ __forceinline__ float exp_neg_kr(float r, float k_hi, float k_lo) {
    const float t = k_hi * r;
    const float t_lo = fmaf(k_lo, r, fmaf(k_hi, r, -t));
    float e;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(-t));
    return e * fmaf(-t_lo, 0.693147182f, 1.0f);
}

// Sum kept as an unevaluated pair hi + lo: Knuth's TwoSum gives the exact
// rounding error of each addition, accumulated in lo (error ~ n eps^2 of the
// sum of magnitudes).
struct TwoFloatSum {
    float hi = 0.0f, lo = 0.0f;
    __device__ __forceinline__ void add(float v) {
        const float t = hi + v;
        const float bp = t - hi;
        lo += (hi - (t - bp)) + (v - bp);
        hi = t;
    }
};

// Kahan (compensated) accumulation: true sum ~= s - c.
__device__ __forceinline__ void kahan_add(float &s, float &c, float v) {
    const float y = v - c;
    const float t = s + y;
    c = (t - s) - y;
    s = t;
}

// ---------------------------------------------------------------------------
// Packed f32x2 arithmetic: one instruction evaluates the same operation for
// two j against one i (sm_100+ FADD2/FMUL2/FFMA2), halving the issue slots
// of the pair arithmetic.  Both halves round exactly like the scalar
// operations.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float2 dup2(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float rsqrt_approx(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// One i particle, each value duplicated into both halves of a pair: hi and
// lo parts of the two-float position (x = xh + xl).
struct PairI {
    float2 xh, yh, xl, yl;
};

// The geometry of i with two j, the j values negated (nxh = -xh_j, ...):
//   dx = x_i - x_j as (xh_i - xh_j) + (xl_i - xl_j) (the hi difference is
//        exact for nearby particles, so dx keeps ~2^-24 of its own size),
//   r2 = dx^2 + dy^2, y = 1/r, ex = e^{-kappa r}.
// 1/r: hardware rsqrt plus one Newton step, which also gives r = r2 y
// refined; e^{-kappa r} = 2^{-(kappa log2 e) r} on the SFU.
__device__ __forceinline__ void pair2_core(const PairI &I, float2 nxh, float2 nyh, float2 nxl, float2 nyl,
                                           float2 nkl2e, float2 &dx, float2 &dy, float2 &r2, float2 &y,
                                           float2 &ex) {
    dx = add2(add2(I.xh, nxh), add2(I.xl, nxl));
    dy = add2(add2(I.yh, nyh), add2(I.yl, nyl));
    r2 = fma2(dx, dx, mul2(dy, dy));
    const float2 y0 = make_float2(rsqrt_approx(r2.x), rsqrt_approx(r2.y));
    const float2 u = mul2(r2, y0);                                  // r, unrefined
    const float2 h = mul2(fma2(u, y0, dup2(-1.0f)), dup2(-0.5f));  // (1 - r2 y0^2) / 2
    y = fma2(h, y0, y0);                                            // 1/r after one Newton step
    const float2 r = fma2(h, u, u);                                 // r = r2 y, from the same step
    const float2 nt = mul2(r, nkl2e);                               // -(kappa log2 e) r
    ex = make_float2(ex2_approx(nt.x), ex2_approx(nt.y));
}

// Pair terms of i with two j (pair2_core), w = q_j e^{-kappa r} y^2 (y +
// kappa), so that the force on i from j is C q_i w (dx, dy) = C q_i q_j (1 +
// kappa r) e^{-kappa r} / r^3 (dx, dy), the reference's pair force
// (ShieldedCoulombForce.cpp:144-157), C q_i applied once per particle.  A
// pair at r2 = 0 gives non-finite w: callers exclude j == i by a select.
__device__ __forceinline__ void pair2_terms(const PairI &I, float2 nxh, float2 nyh, float2 nxl, float2 nyl,
                                            float2 q, float2 kap, float2 nkl2e, float2 &dx, float2 &dy,
                                            float2 &r2, float2 &w) {
    float2 y, ex;
    pair2_core(I, nxh, nyh, nxl, nyl, nkl2e, dx, dy, r2, y, ex);
    w = mul2(mul2(q, ex), mul2(mul2(y, y), add2(y, kap)));
}

// What a sweep reads of its cloud and position set b: of a launch's parameters
// as they are needed (they are constants; held as values they cost the sweep
// registers, 3% on 262,144 particles) ...
struct StageView {
    const StageParams &P;
    int b;
    __device__ __forceinline__ int n() const { return P.c.n; }
    __device__ __forceinline__ const float4 *pa() const { return P.c.pa[b]; }  // packed positions
    __device__ __forceinline__ const float4 *pb() const { return P.c.pb[b]; }
    __device__ __forceinline__ const double *px() const { return P.c.px[b]; }
    __device__ __forceinline__ const double *py() const { return P.c.py[b]; }
    __device__ __forceinline__ const float4 *gbox() const { return P.c.gbox[b]; }
    __device__ __forceinline__ const float4 *gsuper() const { return P.c.gsuper[b]; }
    __device__ __forceinline__ unsigned long long *eval_pairs() const { return P.c.eval_pairs; }
    __device__ __forceinline__ double kappa() const { return P.f.shielding; }
    __device__ __forceinline__ float rc2_lo() const { return P.rc2_lo; }  // these bracket r_c^2: r^2 between
    __device__ __forceinline__ float rc2_hi() const { return P.rc2_hi; }  // them needs the reference's decision
    __device__ __forceinline__ float kappa_f() const { return P.kappa_f; }
    __device__ __forceinline__ float nkl2e() const { return P.nkl2e; }  // -kappa log2(e)
    __device__ __forceinline__ int direct_min() const { return P.direct_min; }
    __device__ __forceinline__ float near_direct_f2() const { return P.near_direct_f2; }
};

// The reference's cutoff decision for particle ii and j = jg; false for j == i
// and where either index is -1 (a lane past the cloud's last particle, which
// sits at the origin and takes part in the direct chunks with the others; a
// padding j).
#pragma nv_exec_check_disable
template <class View>
__host__ __device__ __forceinline__ bool border_in(const View &P, int ii, int jg) {
    if (jg == ii || jg < 0 || ii < 0) return false;
    double r, a;
    return ref_in_cutoff(P.px()[ii] - P.px()[jg], P.py()[ii] - P.py()[jg], P.kappa(), r, a);
}

// The scalar form of one pair for the slow path (pairs within 4e-6 of the
// cutoff in r^2, decided exactly as the reference decides): w as in
// pair2_terms, 0 for a pair outside the cutoff.  j values negated.
template <class View>
__device__ __forceinline__ float border_pair(const View &P, const PairI &I, int ii, float nxh,
                                             float nyh, float nxl, float nyl, float q, int jg, float &dx,
                                             float &dy) {
    dx = (I.xh.x + nxh) + (I.xl.x + nxl);
    dy = (I.yh.x + nyh) + (I.yl.x + nyl);
    if (!border_in(P, ii, jg)) return 0.0f;
    const float r2 = fmaf(dx, dx, dy * dy);
    float y = rsqrt_approx(r2);
    const float u = r2 * y;
    const float h = -0.5f * fmaf(u, y, -1.0f);
    y = fmaf(h, y, y);
    const float rr = fmaf(h, u, u);
    const float ex = ex2_approx(rr * P.nkl2e());
    return (q * ex) * ((y * y) * (y + P.kappa_f()));
}

// Conservative FP32 test: can any point of box a come within the cutoff of
// any point of box b?  Boxes are (x0, y0, x1, y1) of FP32 hi parts; the true
// positions lie within an ulp of them and the box arithmetic rounds, so the
// gaps are shrunk by 2^-20 of the largest coordinate before comparing with
// r_c^2 (already rounded up, rc2_hi).
__device__ __forceinline__ bool boxes_near(const float4 &a, const float4 &b, float rc2_hi) {
    const float gx = fmaxf(a.x - b.z, b.x - a.z);
    const float gy = fmaxf(a.y - b.w, b.y - a.w);
    const float big = fmaxf(fmaxf(fmaxf(fabsf(a.x), fabsf(a.z)), fmaxf(fabsf(b.x), fabsf(b.z))),
                            fmaxf(fmaxf(fabsf(a.y), fabsf(a.w)), fmaxf(fabsf(b.y), fabsf(b.w))));
    const float m = 9.5367431640625e-7f * big;  // 2^-20
    const float dx = fmaxf(0.0f, gx - m), dy = fmaxf(0.0f, gy - m);
    return !(fmaf(dx, dx, dy * dy) >= rc2_hi);  // NaN: near (never drops a pair)
}

// Conservative FP32 test: is every point of box a within the cutoff of every
// point of box b?  The farthest separations are widened by 2^-20 of the
// largest coordinate and the squared distance must stay below 0.999 r_c^2,
// so for every pair of the two groups the reference's FP64 test
// kappa*sqrt(dx*dx + dy*dy) < 10 holds (NaN: false).
__device__ __forceinline__ bool boxes_inside(const float4 &a, const float4 &b, float rc2_lo) {
    const float gx = fmaxf(a.z - b.x, b.z - a.x);
    const float gy = fmaxf(a.w - b.y, b.w - a.y);
    const float big = fmaxf(fmaxf(fmaxf(fabsf(a.x), fabsf(a.z)), fmaxf(fabsf(b.x), fabsf(b.z))),
                            fmaxf(fmaxf(fabsf(a.y), fabsf(a.w)), fmaxf(fabsf(b.y), fabsf(b.w))));
    const float m = 9.5367431640625e-7f * big;  // 2^-20
    const float dx = gx + m, dy = gy + m;
    return fmaf(dx, dx, dy * dy) < 0.999f * rc2_lo;
}

// Barrier `id` of `threads` threads of the block.  The blocks that sweep a
// tile's two position sets hold one half of NW warps per set; each half goes
// through its sweep on its own.
__device__ __forceinline__ void bar_sync(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
constexpr int kBarSet = 1;       // + set: the set's half of the block
constexpr int kBarEpilogue = 3;  // + pair: two warps

// ---------------------------------------------------------------------------
// The j groups within reach of an i tile, by class.  Groups are tested by
// their boxes, 32 consecutive groups (a super group) per warp at a time; in
// large clouds super groups out of reach are skipped whole by their own boxes
// (Morton order keeps both compact), so a tile of a 262,144-particle cloud
// tests 256 + 32 per super group in reach instead of 8192.  The lists keep
// the groups' order.
// ---------------------------------------------------------------------------
constexpr int kSuperCap = 256;  // super groups considered at a time

template <int NW, int NCLASS>
struct NearLists {
    static constexpr int rounds = 16 / NW > 0 ? 16 / NW : 1;  // tests of a warp per batch
    static constexpr int cap = 32 * NW * rounds;              // groups of a batch
    int list[cap];  // the classes one after the other
    int super[kSuperCap];
    int count[NCLASS][NW];
};

// Lists the groups within reach batch by batch and calls use(first, total) for
// every batch that has any (every thread of the NW warps, `tid` its index
// among them): class k's groups are L.list[first[k] .. first[k] + total[k] - 1].
// classify(g, box) is the class of a group within reach.  Of every `stride`
// groups only the `offset`-th is considered (the ranks of a j split share the
// tests); gs: super group boxes (stride 1), or nullptr.
//
// A warp tests its part of a batch on its own and keeps the classes in one
// register per lane; the warps meet twice to lay the lists out.
template <int NW, int NCLASS, class Sync, class Classify, class Use>
__device__ __forceinline__ void for_near_groups(NearLists<NW, NCLASS> &L, const float4 *__restrict__ gb,
                                                const float4 *__restrict__ gs, int ngroups, int offset, int stride,
                                                const float4 &tb, float rc2_hi, int tid, Sync sync, Classify classify,
                                                Use use) {
    constexpr int NR = NearLists<NW, NCLASS>::rounds;
    const int lane = tid & 31, warp = tid >> 5;
    const uint32_t below = (1u << lane) - 1u;
    const int ncand = (ngroups - offset + stride - 1) / stride;  // candidate t is group t*stride + offset
    const int nsuper = (ncand + 31) >> 5;
    for (int s0 = 0; s0 < nsuper; s0 += kSuperCap) {
        int ns = min(kSuperCap, nsuper - s0);
        if (gs) {  // the super groups within reach, in order
            const int all = ns;
            ns = 0;
            for (int t0 = 0; t0 < all; t0 += 32 * NW) {
                const int t = t0 + tid;
                const bool near = t < all && boxes_near(tb, gs[s0 + t], rc2_hi);
                const uint32_t bal = __ballot_sync(0xffffffffu, near);
                if (lane == 0) L.count[0][warp] = __popc(bal);
                sync();
                int off = ns;
#pragma unroll
                for (int w = 0; w < NW; w++) {
                    off += (w < warp) ? L.count[0][w] : 0;
                    ns += L.count[0][w];
                }
                if (near) L.super[off + __popc(bal & below)] = s0 + t;
                sync();
            }
        }
        auto group_of = [&](int e) { return (32 * (gs ? L.super[e] : s0 + e) + lane) * stride + offset; };
        for (int e0 = 0; e0 < ns; e0 += NW * NR) {
            for (int u = 1; u < NR; u++) {  // one round trip to L2 (~900 cycles) for the batch's boxes
                const int e = e0 + u * NW + warp, g = (e < ns) ? group_of(e) : ngroups;
                if (g < ngroups) prefetch_l1(gb + g);
            }
            uint32_t cls = 0u;  // 2 bits per round: class + 1, 0 = out of reach
            static_assert(NR <= 16 && NCLASS <= 3, "classes fit a register");
            int cnt[NCLASS];  // of this warp
#pragma unroll
            for (int k = 0; k < NCLASS; k++) cnt[k] = 0;
            for (int u = 0; u < NR; u++) {
                const int e = e0 + u * NW + warp;
                if (e >= ns) break;
                const int g = group_of(e);
                const float4 box = (g < ngroups) ? gb[g] : make_float4(INFINITY, INFINITY, -INFINITY, -INFINITY);
                const bool near = g < ngroups && boxes_near(tb, box, rc2_hi);
                if (!__any_sync(0xffffffffu, near)) continue;
                const uint32_t c = near ? (uint32_t)classify(g, box) + 1u : 0u;
                cls |= c << (2 * u);
#pragma unroll
                for (int k = 0; k < NCLASS; k++) cnt[k] += __popc(__ballot_sync(0xffffffffu, c == k + 1u));
            }
            if (lane == 0)
#pragma unroll
                for (int k = 0; k < NCLASS; k++) L.count[k][warp] = cnt[k];
            sync();
            int first[NCLASS], total[NCLASS], off[NCLASS], at = 0;
#pragma unroll
            for (int k = 0; k < NCLASS; k++) {
                first[k] = off[k] = at;
#pragma unroll
                for (int w = 0; w < NW; w++) {
                    off[k] += (w < warp) ? L.count[k][w] : 0;
                    at += L.count[k][w];
                }
                total[k] = at - first[k];
            }
            if (at == 0) {
                sync();  // the counts are rewritten
                continue;
            }
            for (int u = 0; u < NR; u++) {
                const int e = e0 + u * NW + warp;
                const uint32_t c = (cls >> (2 * u)) & 3u;
                if (!__any_sync(0xffffffffu, c != 0u)) continue;
                const int g = group_of(e);
#pragma unroll
                for (int k = 0; k < NCLASS; k++) {
                    const uint32_t bal = __ballot_sync(0xffffffffu, c == k + 1u);
                    if (c == k + 1u) L.list[off[k] + __popc(bal & below)] = g;
                    off[k] += __popc(bal);
                }
            }
            sync();
            use(first, total);
            sync();
        }
    }
}

// ---------------------------------------------------------------------------
// FP32-compensated kernel.
//
// A CTA of NW warps shares one i tile of 32*ILP particles (lane l, slot k ->
// i = tile*32*ILP + k*32 + l).  Each staged j chunk (4 j) goes to one warp;
// its pairs are classified:
//   * groups entirely within the cutoff of the tile (box test): evaluated
//     directly, every lane on the same j from shared-memory broadcasts, two
//     j per packed instruction, no filter and no cutoff test;
//   * other groups within reach: the packed filter on all 4 j and every
//     slot, each lane recording its own passing j as hit bits (a funnel shift
//     of the sign per pair; 8 chunks per 32-bit word); per word and slot the
//     number of (lane, j) pairs that passed decides (a warp reduction): at
//     least 8 P.direct_min of the 1024 -> the 8 chunks are evaluated directly
//     for that slot with the cutoff taken by a select; fewer -> each lane
//     evaluates its hits of the whole staged tile two at a time.
// Each lane accumulates only into its own sums (plain f32x2 sums over a few
// chunks, then Kahan), so the result is deterministic and needs no atomics.
// The sums leave out C q_i (applied in FP64 once per particle).
// ---------------------------------------------------------------------------
template <int NW, int ILP, int TC>
struct Fp32cSmem {
    // j tile: TC 4-j chunks, each field of the 4 j in one 16-byte word
    // (-xh, -yh, |p|^2, -xl, -yl, q, j): two consecutive j of a field load
    // straight into the register pair a packed instruction takes
    static constexpr size_t tile = (size_t)TC * 7 * sizeof(float4);
    static constexpr size_t cold = (size_t)ILP * 32 * sizeof(float4);
    static constexpr size_t acc = (size_t)NW * ILP * 32 * sizeof(float4);
    static constexpr size_t red = (size_t)ILP * 32 * sizeof(float4);
    // culling: near, inside and mostly-inside group lists
    static constexpr size_t glist = sizeof(NearLists<NW, 3>);
    static constexpr size_t bytes = tile + cold + acc + red + glist;
    // s_red, in float4 units from the start of shared memory
    static constexpr size_t red_offset = (tile + cold + acc) / sizeof(float4);
};

// The FP32C sweep of one i tile against rank `rank` of S of the j chunks:
// of the view's position set: i-side setup, the classified j loop, and the combine of the NW warps'
// Kahan sums into s_red[TILE] = (sx, sy, cx, cy) (force / (C q_i) = s - c).
// By NW warps (`tid` the thread's index among them, sync() their barrier); ends
// with them synchronised.  `P` may live in shared memory (batched
// kernel).  j at or beyond n read as
// padding, so a cloud needs no padding of its own.
template <int NW, int ILP, int TC, bool CULL, class View, class Sync>
__device__ __forceinline__ void fp32c_sweep(const View &P, int tile, int rank, int S, int tid, Sync sync,
                                            unsigned char *smem_raw) {
    constexpr int NT = NW * 32;
    constexpr int TILE = 32 * ILP;  // particles per i tile
    static_assert(ILP <= 4, "the i slots of a lane are selected with unrolled compares");
    float4 *s_x4 = reinterpret_cast<float4 *>(smem_raw);  // [TC] -xh of 4 j
    float4 *s_y4 = s_x4 + TC;                              // [TC] -yh
    float4 *s_b4 = s_y4 + TC;                              // [TC] xh^2 + yh^2
    float4 *s_xl4 = s_b4 + TC;                             // [TC] -xl
    float4 *s_yl4 = s_xl4 + TC;                            // [TC] -yl
    float4 *s_q4 = s_yl4 + TC;                             // [TC] q
    int4 *s_j4 = reinterpret_cast<int4 *>(s_q4 + TC);      // [TC] j (-1: padding)
    float4 *s_cold = reinterpret_cast<float4 *>(s_j4 + TC);  // [ILP][32] (xl, yl, -, i)
    float4 *s_acc = s_cold + ILP * 32;                     // [NW][ILP][32]
    float4 *s_red = s_acc + NW * ILP * 32;                 // [TILE]

    const int lane = tid & 31, warp = tid >> 5;
    const int n = P.n();
    const float4 *__restrict__ pa = P.pa();
    const float4 *__restrict__ pb = P.pb();
    float4 *my_acc = s_acc + warp * ILP * 32;
    const float2 kap = dup2(P.kappa_f()), nkl2e = dup2(P.nkl2e());
    const float rc2_lo = P.rc2_lo(), rc2_hi = P.rc2_hi();

    // every warp owns the same TILE particles: lane l, slot k -> i = tile*TILE + k*32 + l.
    // i side duplicated into both halves of a packed pair: the packed FMAs
    // evaluate two consecutive j against one i
    float2 px2[ILP], py2[ILP], nu2[ILP];  // 2 xh_i, 2 yh_i, -(filter bound)
#pragma unroll
    for (int k = 0; k < ILP; k++) {
        const int i = tile * TILE + k * 32 + lane;
        float ax = 0.0f, ay = 0.0f, nu = INFINITY;
        float4 cold = make_float4(0.0f, 0.0f, 0.0f, __int_as_float(-1));
        if (i < n) {
            const float4 A = pa[i];
            const float4 B = pb[i];
            ax = A.x;
            ay = A.y;
            nu = B.z;
            cold = make_float4(B.x, B.y, 0.0f, __int_as_float(i));
        }
        px2[k] = dup2(2.0f * ax);
        py2[k] = dup2(2.0f * ay);
        nu2[k] = dup2(nu);
        if (warp == 0) s_cold[k * 32 + lane] = cold;
        my_acc[k * 32 + lane] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    // i side of slot k (runtime k: the slow paths exist once in the code)
    auto slot_i = [&](int k, int &ii) {
        float xh = 0.5f * px2[0].x, yh = 0.5f * py2[0].x;
#pragma unroll
        for (int t = 1; t < ILP; t++) {
            xh = (k == t) ? 0.5f * px2[t].x : xh;
            yh = (k == t) ? 0.5f * py2[t].x : yh;
        }
        const float4 c4 = s_cold[k * 32 + lane];
        ii = __float_as_int(c4.w);
        return PairI{dup2(xh), dup2(yh), dup2(c4.x), dup2(c4.y)};
    };

    // Filter hits are recorded per lane, one word per 8 chunks this warp swept:
    // bit 31 - (4 g + u) of word w of slot k is the pair (slot k's i, j = 4 (warp
    // + (8 w + g) NW) + u of the staged tile).  A tile holds at most kWords
    // words of a warp's chunks; they are evaluated together, every lane its own
    // hits two at a time, so a lane with few hits in one stretch of j makes up
    // for it in another (0.5 hits per lane and word on a calm cloud: word by
    // word, five of six lanes were idle).
    constexpr int kWords = (TC / NW + 7) / 8;
    const float *s_xf = reinterpret_cast<const float *>(s_x4);
    const float *s_yf = reinterpret_cast<const float *>(s_y4);
    const float *s_xlf = reinterpret_cast<const float *>(s_xl4);
    const float *s_ylf = reinterpret_cast<const float *>(s_yl4);
    const float *s_qf = reinterpret_cast<const float *>(s_q4);
    const int *s_jf = reinterpret_cast<const int *>(s_j4);
    auto flush_hits = [&](int k, uint32_t (&m)[kWords]) {
        int ii;
        const PairI I = slot_i(k, ii);
        float4 acc = my_acc[k * 32 + lane];
        // the next hit's index into the tile's j; words in order
        auto next = [&]() {
            int w = 0;
            uint32_t v = m[0];
#pragma unroll
            for (int t = 1; t < kWords; t++)
                if (v == 0u) {
                    v = m[t];
                    w = t;
                }
            const int pos = __clz(v);
            v &= ~(0x80000000u >> pos);
#pragma unroll
            for (int t = 0; t < kWords; t++) m[t] = (t == w) ? v : m[t];
            return 4 * (warp + (8 * w + (pos >> 2)) * NW) + (pos & 3);
        };
        auto any = [&]() {
            uint32_t v = 0u;
#pragma unroll
            for (int t = 0; t < kWords; t++) v |= m[t];
            return v != 0u;
        };
        while (any()) {
            // two hits per packed evaluation; a missing second one repeats
            // the first with q = 0 (a finite, zero term)
            const int j0 = next();
            const bool two = any();
            const int j1 = two ? next() : j0;
            const float q1 = two ? 1.0f : 0.0f;
            float2 dx, dy, r2, w;
            pair2_terms(I, make_float2(s_xf[j0], s_xf[j1]), make_float2(s_yf[j0], s_yf[j1]),
                        make_float2(s_xlf[j0], s_xlf[j1]), make_float2(s_ylf[j0], s_ylf[j1]),
                        make_float2(s_qf[j0], s_qf[j1] * q1), kap, nkl2e, dx, dy, r2, w);
            const int g0 = s_jf[j0], g1 = s_jf[j1];
            // certainly inside: r2 < rc2_lo; borderline pairs decided exactly
            w.x = (r2.x < rc2_lo && g0 != ii) ? w.x : 0.0f;
            w.y = (r2.y < rc2_lo && g1 != ii && two) ? w.y : 0.0f;
            if (!(r2.x < rc2_lo) && r2.x < rc2_hi) {
                float bx, by;
                w.x = border_pair(P, I, ii, s_xf[j0], s_yf[j0], s_xlf[j0], s_ylf[j0], s_qf[j0], g0, bx, by);
            }
            if (two && !(r2.y < rc2_lo) && r2.y < rc2_hi) {
                float bx, by;
                w.y = border_pair(P, I, ii, s_xf[j1], s_yf[j1], s_xlf[j1], s_ylf[j1], s_qf[j1], g1, bx, by);
            }
            const float2 fx = mul2(w, dx), fy = mul2(w, dy);
            kahan_add(acc.x, acc.z, fx.x + fx.y);
            kahan_add(acc.y, acc.w, fy.x + fy.y);
        }
        my_acc[k * 32 + lane] = acc;
    };

    // Chunk c of the staged tile against slot k (runtime k), every lane on
    // the same 4 j, the cutoff taken by a select (pairs within 4e-6 of it in
    // r^2 decided exactly, j == i excluded); the chunk's terms summed plainly
    // and added to the slot's compensated sums.
    const int tile_j0 = tile * TILE;  // the tile's own particles: the only chunks that can hold j == i
    auto direct_chunk = [&](int c, int k) {
        int ii;
        const PairI I = slot_i(k, ii);
        const float4 X = s_x4[c], Y = s_y4[c], XL = s_xl4[c], YL = s_yl4[c], Q = s_q4[c];
        float2 dx, dy, r2, w, dx2, dy2, r22, w2;
        pair2_terms(I, make_float2(X.x, X.y), make_float2(Y.x, Y.y), make_float2(XL.x, XL.y),
                    make_float2(YL.x, YL.y), make_float2(Q.x, Q.y), kap, nkl2e, dx, dy, r2, w);
        pair2_terms(I, make_float2(X.z, X.w), make_float2(Y.z, Y.w), make_float2(XL.z, XL.w),
                    make_float2(YL.z, YL.w), make_float2(Q.z, Q.w), kap, nkl2e, dx2, dy2, r22, w2);
        if ((unsigned)(s_jf[4 * c] - tile_j0) < (unsigned)TILE) {  // warp-uniform: this tile's own chunk
            const int4 J = s_j4[c];
            w.x = (r2.x < rc2_lo && J.x != ii) ? w.x : 0.0f;
            w.y = (r2.y < rc2_lo && J.y != ii) ? w.y : 0.0f;
            w2.x = (r22.x < rc2_lo && J.z != ii) ? w2.x : 0.0f;
            w2.y = (r22.y < rc2_lo && J.w != ii) ? w2.y : 0.0f;
        } else {
            w.x = (r2.x < rc2_lo) ? w.x : 0.0f;
            w.y = (r2.y < rc2_lo) ? w.y : 0.0f;
            w2.x = (r22.x < rc2_lo) ? w2.x : 0.0f;
            w2.y = (r22.y < rc2_lo) ? w2.y : 0.0f;
        }
        const bool bd = (!(r2.x < rc2_lo) && r2.x < rc2_hi) || (!(r2.y < rc2_lo) && r2.y < rc2_hi) ||
                        (!(r22.x < rc2_lo) && r22.x < rc2_hi) || (!(r22.y < rc2_lo) && r22.y < rc2_hi);
        float2 fx = fma2(w2, dx2, mul2(w, dx));
        float2 fy = fma2(w2, dy2, mul2(w, dy));
        if (bd) {  // rare: pairs within 4e-6 of the cutoff in r^2
#pragma unroll 1
            for (int u = 0; u < 4; u++) {
                const float rr = (u == 0) ? r2.x : (u == 1) ? r2.y : (u == 2) ? r22.x : r22.y;
                if (rr < rc2_lo || !(rr < rc2_hi)) continue;
                const int jj = 4 * c + u;
                float bx, by;
                const float wb = border_pair(P, I, ii, s_xf[jj], s_yf[jj], s_xlf[jj], s_ylf[jj], s_qf[jj],
                                             s_jf[jj], bx, by);
                fx.x = fmaf(wb, bx, fx.x);
                fy.x = fmaf(wb, by, fy.x);
            }
        }
        float4 acc = my_acc[k * 32 + lane];
        kahan_add(acc.x, acc.z, fx.x + fx.y);
        kahan_add(acc.y, acc.w, fy.x + fy.y);
        my_acc[k * 32 + lane] = acc;
    };

    // Sweeps the `count` chunks (4 consecutive j) of this CTA's list through
    // shared-memory tiles; chunk_of(q) is the cloud chunk index of entry q.
    // Within a tile, chunk c goes to warp c % NW.
    // MODE 0: the packed filter, then direct chunks or hit bits; 1: groups
    // entirely inside the cutoff; 2: groups mostly inside it, every chunk
    // evaluated directly with the cutoff taken by a select (no filter)
    auto sweep = [&](int count, auto chunk_of, auto mode_tag) {
    constexpr int MODE = decltype(mode_tag)::value;
    constexpr bool DENSE = MODE == 1;
    for (int q0 = 0; q0 < count; q0 += TC) {
        const int tcn = min(TC, count - q0);
        sync();
        for (int e = tid; e < tcn; e += NT) {
            const int jb = 4 * chunk_of(q0 + e);  // first j of the chunk
            float xs[4], ys[4], bs[4];
            float *xl = reinterpret_cast<float *>(s_xl4 + e), *yl = reinterpret_cast<float *>(s_yl4 + e);
            float *qs = reinterpret_cast<float *>(s_q4 + e);
            int *js = reinterpret_cast<int *>(s_j4 + e);
#pragma unroll
            for (int u = 0; u < 4; u++) {
                if (jb + u < n) {
                    const float4 A = pa[jb + u];
                    const float4 B = pb[jb + u];
                    xs[u] = -A.x;
                    ys[u] = -A.y;
                    bs[u] = A.z;
                    xl[u] = -B.x;
                    yl[u] = -B.y;
                    qs[u] = A.w;
                    js[u] = jb + u;
                } else {  // padding: never passes the filter; a finite, zero term
                    xs[u] = -kPadPosition;
                    ys[u] = -kPadPosition;
                    bs[u] = INFINITY;
                    xl[u] = yl[u] = qs[u] = 0.0f;
                    js[u] = -1;
                }
            }
            s_x4[e] = make_float4(xs[0], xs[1], xs[2], xs[3]);
            s_y4[e] = make_float4(ys[0], ys[1], ys[2], ys[3]);
            s_b4[e] = make_float4(bs[0], bs[1], bs[2], bs[3]);
        }
        sync();
        if constexpr (DENSE) {
            // every pair of these groups is inside the cutoff (and j != i):
            // no filter, no select; each lane evaluates its own i against the
            // chunk's 4 j, two per packed instruction, its i data and sums in
            // registers for the whole tile; plain sums over two chunks, then Kahan
            PairI I[ILP];
            float4 acc[ILP];
            float2 fx[ILP], fy[ILP];
#pragma unroll
            for (int k = 0; k < ILP; k++) {
                int ii;
                I[k] = slot_i(k, ii);
                acc[k] = my_acc[k * 32 + lane];
                fx[k] = fy[k] = dup2(0.0f);
            }
            int ng = 0;
            for (int c = warp; c < tcn; c += NW) {
                const float4 X = s_x4[c], Y = s_y4[c], XL = s_xl4[c], YL = s_yl4[c], Q = s_q4[c];
#pragma unroll
                for (int k = 0; k < ILP; k++) {
                    float2 dx, dy, r2, w;
                    pair2_terms(I[k], make_float2(X.x, X.y), make_float2(Y.x, Y.y), make_float2(XL.x, XL.y),
                                make_float2(YL.x, YL.y), make_float2(Q.x, Q.y), kap, nkl2e, dx, dy, r2, w);
                    fx[k] = fma2(w, dx, fx[k]);
                    fy[k] = fma2(w, dy, fy[k]);
                    pair2_terms(I[k], make_float2(X.z, X.w), make_float2(Y.z, Y.w), make_float2(XL.z, XL.w),
                                make_float2(YL.z, YL.w), make_float2(Q.z, Q.w), kap, nkl2e, dx, dy, r2, w);
                    fx[k] = fma2(w, dx, fx[k]);
                    fy[k] = fma2(w, dy, fy[k]);
                }
                if (++ng == 2) {
                    ng = 0;
#pragma unroll
                    for (int k = 0; k < ILP; k++) {
                        kahan_add(acc[k].x, acc[k].z, fx[k].x + fx[k].y);
                        kahan_add(acc[k].y, acc[k].w, fy[k].x + fy[k].y);
                        fx[k] = fy[k] = dup2(0.0f);
                    }
                }
            }
#pragma unroll
            for (int k = 0; k < ILP; k++) {
                kahan_add(acc[k].x, acc[k].z, fx[k].x + fx[k].y);
                kahan_add(acc[k].y, acc[k].w, fy[k].x + fy[k].y);
                my_acc[k * 32 + lane] = acc[k];
            }
        } else if constexpr (MODE == 2) {
            for (int c = warp; c < tcn; c += NW) {
#pragma unroll 1
                for (int k = 0; k < ILP; k++) direct_chunk(c, k);
            }
        } else {
            uint32_t hits[ILP][kWords];
#pragma unroll
            for (int w = 0; w < kWords; w++) {
                uint32_t m[ILP];
#pragma unroll
                for (int k = 0; k < ILP; k++) m[k] = 0u;
                const int c0 = warp + 8 * w * NW, gn = min(8, (tcn - c0 + NW - 1) / NW);  // this word's chunks
                if (gn <= 0) {  // warp-uniform: the tile is done
#pragma unroll
                    for (int k = 0; k < ILP; k++) hits[k][w] = 0u;
                    continue;
                }
#pragma unroll 2
                for (int g = 0; g < gn; g++) {
                    const int c = c0 + g * NW;
                    const float4 X = s_x4[c], Y = s_y4[c], Bq = s_b4[c];
                    const float2 X01 = make_float2(X.x, X.y), X23 = make_float2(X.z, X.w);
                    const float2 Y01 = make_float2(Y.x, Y.y), Y23 = make_float2(Y.z, Y.w);
                    const float2 B01 = make_float2(Bq.x, Bq.y), B23 = make_float2(Bq.z, Bq.w);
                    // d = |p_j|^2 - 2 p_i.p_j - bound_i: pair (i, j) passes iff d < 0
#pragma unroll
                    for (int k = 0; k < ILP; k++) {
                        const float2 d01 = fma2(px2[k], X01, fma2(py2[k], Y01, add2(B01, nu2[k])));
                        const float2 d23 = fma2(px2[k], X23, fma2(py2[k], Y23, add2(B23, nu2[k])));
                        m[k] = __funnelshift_l(__float_as_uint(d01.x), m[k], 1);
                        m[k] = __funnelshift_l(__float_as_uint(d01.y), m[k], 1);
                        m[k] = __funnelshift_l(__float_as_uint(d23.x), m[k], 1);
                        m[k] = __funnelshift_l(__float_as_uint(d23.y), m[k], 1);
                    }
                }
                // enough passing (lane, j) pairs: the word's chunks directly
#pragma unroll
                for (int k = 0; k < ILP; k++) {
                    if (gn < 8) m[k] <<= 32 - 4 * gn;
                    if ((int)__reduce_add_sync(0xffffffffu, __popc(m[k])) >= 8 * P.direct_min()) {
#pragma unroll 1
                        for (int g = 0; g < gn; g++) direct_chunk(c0 + g * NW, k);
                        m[k] = 0u;
                    }
                    hits[k][w] = m[k];
                }
            }
#pragma unroll 1
            for (int k = 0; k < ILP; k++) {
                uint32_t m[kWords], v = 0u;
#pragma unroll
                for (int w = 0; w < kWords; w++) {
                    m[w] = hits[0][w];
#pragma unroll
                    for (int t = 1; t < ILP; t++) m[w] = (k == t) ? hits[t][w] : m[w];
                    v |= m[w];
                }
                if (__any_sync(0xffffffffu, v != 0u)) flush_hits(k, m);
            }
        }
    }
    };

    sync();  // s_cold complete
    if constexpr (!CULL) {
        // chunks dealt round-robin: chunk c belongs to rank c % S, so every
        // rank (and every warp) samples the whole cloud evenly
        const int nch_all = (n + 3) >> 2;
        const int my_nch = (nch_all - rank + S - 1) / S;  // chunks of this rank
        sweep(my_nch, [&](int q) { return q * S + rank; }, std::integral_constant<int, 0>{});
    } else {
        // the 32-particle groups whose box is within the cutoff of the tile's
        // box (the others hold no pair the reference counts), dealt
        // round-robin to the ranks, class by class
        const float4 *__restrict__ gb = P.gbox();
        NearLists<NW, 3> &L = *reinterpret_cast<NearLists<NW, 3> *>(s_red + TILE);
        const int ngroups = (n + 31) >> 5;
        float4 tb = gb[tile * ILP];
#pragma unroll
        for (int k = 1; k < ILP; k++) {
            if (tile * ILP + k < ngroups) {  // a cloud's last tile may hold fewer groups
                const float4 v = gb[tile * ILP + k];
                tb = make_float4(fminf(tb.x, v.x), fminf(tb.y, v.y), fmaxf(tb.z, v.z), fmaxf(tb.w, v.w));
            }
        }
        unsigned long long swept = 0ull;
        const float rc2_mostly = P.rc2_lo() * P.near_direct_f2();  // 0: no such class
        const float4 *gs = P.gsuper();
        // the ranks share the tests (rank r takes every S-th group), or, with
        // super groups, the groups found
        const int deal = gs ? S : 1, mine_of = gs ? rank : 0;
        for_near_groups(
            L, gb, gs, ngroups, gs ? 0 : rank, gs ? 1 : S, tb, P.rc2_hi(), tid, sync,
            [&](int g, const float4 &gbox) {
                // the tile's own groups hold the pairs j == i: not "inside"
                if (g / ILP != tile && boxes_inside(tb, gbox, P.rc2_lo())) return 1;
                // farthest separation within sqrt(near_direct_f2) r_c: most
                // pairs pass the filter, so it is skipped
                return (rc2_mostly > 0.0f && boxes_inside(tb, gbox, rc2_mostly)) ? 2 : 0;
            },
            [&](const int (&first)[3], const int (&total)[3]) {
                auto mine = [&](int t) { return 8 * ((t - mine_of + deal - 1) / deal); };  // this rank's chunks of t groups
                auto chunk_of = [&](int k, int q) { return 8 * L.list[first[k] + (q >> 3) * deal + mine_of] + (q & 7); };
                sweep(mine(total[0]), [&](int q) { return chunk_of(0, q); }, std::integral_constant<int, 0>{});
                sweep(mine(total[1]), [&](int q) { return chunk_of(1, q); }, std::integral_constant<int, 1>{});
                sweep(mine(total[2]), [&](int q) { return chunk_of(2, q); }, std::integral_constant<int, 2>{});
                swept += (unsigned long long)(total[0] + total[1] + total[2]);
            });
        if (tid == 0 && (rank == 0 || !gs) && swept)
            atomicAdd(P.eval_pairs(), swept * 32ull * (unsigned long long)TILE);
    }

    // combine the NW warps in fixed order with a compensated FP32 sum (each
    // warp's Kahan pair (s, c) stands for s - c); FP64 comes later, once per
    // particle (FP64 runs at 1/64 of the FP32 rate here)
    sync();
    for (int e = tid; e < TILE; e += NT) {
        float sx = 0.0f, cx = 0.0f, sy = 0.0f, cy = 0.0f;
#pragma unroll
        for (int w = 0; w < NW; w++) {
            const float4 v = s_acc[w * ILP * 32 + e];
            kahan_add(sx, cx, v.x);
            kahan_add(sx, cx, -v.z);
            kahan_add(sy, cy, v.y);
            kahan_add(sy, cy, -v.w);
        }
        s_red[e] = make_float4(sx, sy, cx, cy);
    }
    sync();
}

// C q_i in FP64: the factor the sweeps leave out of their sums.
__device__ __forceinline__ double pair_scale(const StageParams &P, int i) {
    return __dmul_rn(P.coulomb, P.c.q[i]);
}

// ---------------------------------------------------------------------------
// The epilogue of a pass for one 32-particle group, by two warps.
// ---------------------------------------------------------------------------

struct EpilogueShared {
    double v[2][32];  // [axis][particle]: the velocities of the second set's force
    union {
        struct {
            float hi[2][2][32], lo[2][2][32];  // [set][axis][particle]
        };
        PositionTerms terms[2][32];  // [set][particle]
    };
};

// What the epilogue needs to know of a particle's cloud (a batch holds many).
struct EpilogueCloud {
    const ForceParams &f;
    float rc2_up;
    bool live;  // the lane holds a particle
    int group;  // its 32-particle group among the cloud's (batch's) boxes
};

// Starts bringing the operands of pass_epilogue for particle i, axis ax, into L1.
__device__ __forceinline__ void epilogue_prefetch(const StageParams &P, int i, int ax) {
    const CloudDev &c = P.c;
    prefetch_l1((ax ? c.y : c.x) + i);
    prefetch_l1((ax ? c.vy : c.vx) + i);
    prefetch_l1(c.q + i);
    prefetch_l1(c.m + i);
    prefetch_l1(c.invm + i);
    prefetch_l1(c.orig + i);
    if (P.mode == kModeForceOnly) return;
    if (P.pass == 0) {
        prefetch_l1((ax ? c.py : c.px)[1] + i);
    } else {
        prefetch_l1((ax ? c.py : c.px)[2] + i);
        prefetch_l1((ax ? c.py : c.px)[3] + i);
        prefetch_l1(c.k1[ax] + i);
        prefetch_l1(c.k2[ax] + i);
    }
}

// One axis of particle i's part of the pass, the total force at set e and
// axis velocity v given by force(e, x, v): the new positions of both sets
// (out[0], out[1]), stored but for their packed words; returns whether the
// positions are finite.  Lanes that are not live (i any particle) store nothing.
template <class Force>
__device__ __forceinline__ bool advance_axis(const StageParams &P, int i, int ax, bool live, double (&out)[2],
                                             Force force) {
    const CloudDev &c = P.c;
    double *X = ax ? c.y : c.x, *V = ax ? c.vy : c.vx;
    double *const *p = ax ? c.py : c.px;
    const double dt = stage_dt(P), m = c.m[i];
    const double x = X[i], v = V[i], inv = c.invm[i];
    auto increment = [&](double F) { return div_by(__dmul_rn(dt, F), m, inv); };
    bool fine = true;
    double k1, k2, v2;
    if (P.pass == 0) {
        const double x2 = p[1][i];
        k1 = increment(force(0, x, v));
        v2 = half_step(v, k1);
        k2 = increment(force(1, x2, v2));
        fine = finite64(x2);
    } else {
        k1 = c.k1[ax][i];
        k2 = c.k2[ax][i];
        v2 = half_step(v, k1);
    }
    const double l2 = __dmul_rn(dt, v2);
    if (P.order == 2) {  // x += l2, V += k2; the positions go to sets 2 and 3 (see adopt_sets)
        const double vn = __dadd_rn(v, k2);
        out[0] = __dadd_rn(x, l2);
        out[1] = half_step(out[0], __dmul_rn(dt, vn));
        if (live) {
            V[i] = vn;
            p[2][i] = out[0];
            p[3][i] = out[1];
        }
        return fine && finite64(out[0]);
    }
    const double v3 = half_step(v, k2), l3 = __dmul_rn(dt, v3);
    if (P.pass == 0) {
        out[0] = half_step(x, l2);
        out[1] = __dadd_rn(x, l3);
        if (live) {
            c.k1[ax][i] = k1;
            c.k2[ax][i] = k2;
            p[2][i] = out[0];
            p[3][i] = out[1];
        }
        return fine && finite64(out[0]) && finite64(out[1]);
    }
    const double k3 = increment(force(0, p[2][i], v3));
    const double v4 = __dadd_rn(v, k3);
    const double k4 = increment(force(1, p[3][i], v4));
    const double xn = rk4_sum(x, __dmul_rn(dt, v), l2, l3, __dmul_rn(dt, v4));
    const double vn = rk4_sum(v, k1, k2, k3, k4);
    out[0] = xn;
    out[1] = half_step(xn, __dmul_rn(dt, vn));  // the next step's x2, for the same dt
    if (live) {
        X[i] = xn;
        V[i] = vn;
        p[1][i] = out[1];
    }
    return finite64(xn);
}

// The pass's epilogue for one 32-particle group: lane = particle i, warp ax =
// 0 or 1 of the two computes that axis (they meet at named barrier `bar`);
// fs0, fs1 the pair forces along it at the two sets, C q_i included.  Sums the
// forces, advances the particles, writes the next pass's position sets and
// their group boxes (force-only: the forces, in the caller's order).
//
// The epilogue is a chain of dependent FP64 operations at 64 cycles each; two
// axes are two chains.  The forces outside kBasicForces couple the axes: their
// position terms are computed first (TERMS: the caller has done so), a set per
// warp, and before the second set's force the warps exchange their velocities.
template <bool TERMS = false>
__device__ __forceinline__ void pass_epilogue(const StageParams &P, const EpilogueCloud &E, int i, int ax, int bar,
                                              double fs0, double fs1, EpilogueShared &S) {
    const int lane = threadIdx.x & 31;
    const CloudDev &c = P.c;
    const ForceParams &f = E.f;
    const bool live = E.live;
    const bool fo = P.mode == kModeForceOnly;
    const bool basic = !(f.flags & ~kBasicForces);
    auto meet = [&] { bar_sync(bar, 64); };
    const int ob = (P.pass == 0) ? 2 : 0;  // first buffer written
    if (!basic && !TERMS) {
        if (live && ax < P.nsets) {
            const int b = P.buf[ax];
#pragma unroll
            for (int part = 0; part < kTermParts; part++)
                position_terms(S.terms[ax][lane], part, f, c.px[b][i], c.py[b][i], c.q[i],
                               (f.flags & kDriving) ? stage_time(P, ax) : 0.0);
        }
        meet();
    }
    double out[2] = {0.0, 0.0};
    const int j = live ? i : 0;  // lanes without a particle take part in the meetings
    const double q = c.q[j], m = c.m[j];
    auto force = [&](int e, double x, double v) {
        const double fp = e ? fs1 : fs0;
        if (basic) {
            double therm = 0.0;
            if (f.flags & kThermal) {
                const double2 t = stage_thermal(P, f, j, e);
                therm = ax ? t.y : t.x;
            }
            return axis_force(f, ax, x, v, q, m, fp, therm);
        }
        double vo;  // the other axis's velocity
        if (e == 0) {
            vo = (ax ? c.vx : c.vy)[j];
            if (!fo && P.pass == 1) vo = half_step(vo, c.k2[1 - ax][j]);
        } else {
            S.v[ax][lane] = v;
            meet();
            vo = S.v[1 - ax][lane];
        }
        const int b = P.buf[e];
        const ParticleAt s{c.px[b][j], c.py[b][j], ax ? vo : v, ax ? v : vo, q, m};
        return total_force(P, f, j, e, ax, s, S.terms[e][lane], fp);
    };
    if (fo) {
        const double F = force(0, (ax ? c.py : c.px)[P.buf[0]][j], (ax ? c.vy : c.vx)[j]);
        if (live) (ax ? P.fy_out : P.fx_out)[c.orig[i]] = F;
        return;  // uniform over the launch
    }
    if (!advance_axis(P, j, ax, live, out, force) && live) atomicOr(c.err, 1);
    if (!basic) meet();  // the terms' memory is used again
#pragma unroll
    for (int e = 0; e < 2; e++) {
        float h = 0.0f, lo = 0.0f;
        if (live) split2(out[e], h, lo);
        S.hi[e][ax][lane] = h;
        S.lo[e][ax][lane] = lo;
    }
    meet();
    // write_stage_position's packed words and the group's box, one set per warp
    const int e = ax;
    const float xh = S.hi[e][0][lane], yh = S.hi[e][1][lane];
    if (live) {
        c.pa[ob + e][i] = make_float4(xh, yh, fmaf(yh, yh, xh * xh), c.pa[P.buf[0]][i].w);
        c.pb[ob + e][i] = make_float4(S.lo[e][0][lane], S.lo[e][1][lane], -filter_threshold(xh, yh, E.rc2_up), 0.0f);
    }
    store_group_box(c.gbox[ob + e] + E.group, live, xh, yh, true);
}

// ---------------------------------------------------------------------------
// FP32C pair kernel.
//
// CL = true: a block holds NW warps per position set of the launch, the S
// ranks of a tile form a thread-block cluster, combine through distributed
// shared memory and run the epilogue in the same launch.  CL = false: plain
// blocks of NW warps for one set; each writes its partial sums to global
// memory and stage_finish (below) completes the pass.
// Occupancy: with two i slots per lane the kernel is bounded to 64
// registers, so 32 warps per SM are resident (more latency hidden in the
// sparse phases, where a block is short and bound by dependent loads and
// barriers); four slots need more registers and stay at 24 warps.
// ---------------------------------------------------------------------------
template <int NW, int ILP>
constexpr int fp32c_min_blocks() {
    return (ILP <= 2 ? 32 : 24) / NW > 0 ? (ILP <= 2 ? 32 : 24) / NW : 1;
}

// The epilogue of a tile: pairs of warps of the first block take its groups
// in turn, adding the S ranks' sums (s_red of each set, `stride` float4 apart)
// in order.  The first pair is the tile's number modulo the pairs: warp w
// issues on scheduler w mod 4, and each scheduler has an FP64 unit of its own.
template <int ILP>
__device__ __forceinline__ void tile_epilogue(const StageParams &P, float4 *s_red, int stride, int tile, int S,
                                              EpilogueShared *shared) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int npairs = blockDim.x >> 6, pair = ((warp >> 1) + tile) % npairs;
    const int ax = warp & 1;
#pragma unroll 1
    for (int g = pair; g < ILP; g += npairs) {
        const int e = g * 32 + lane, i = tile * 32 * ILP + e;
        double f[2] = {0.0, 0.0};
        const double cq = (i < P.c.n) ? pair_scale(P, i) : 0.0;
        for (int set = 0; set < P.nsets; set++) {
            float4 *mine = s_red + set * stride + e;
            float4 v = *mine;
            TwoFloatSum sum;
            sum.add(ax ? v.y : v.x);
            float lost = ax ? v.w : v.z;
            for (int r = 1; r < S; r++) {
                v = *cg::this_cluster().map_shared_rank(mine, r);
                sum.add(ax ? v.y : v.x);
                lost += ax ? v.w : v.z;
            }
            f[set] = __dmul_rn(cq, widen(sum.hi) + widen(sum.lo - lost));
        }
        pass_epilogue(P, EpilogueCloud{P.f, P.c.rc2_up, i < P.c.n, i >> 5}, i, ax, kBarEpilogue + (warp >> 1), f[0],
                      f[1], shared[g]);
    }
}

template <int NW, int ILP, int TC, bool CL, bool CULL = false>
__global__ void __launch_bounds__((CL ? 2 : 1) * NW * 32, fp32c_min_blocks<(CL ? 2 : 1) * NW, ILP>())
    pair_stage_fp32c(const StageParams P) {
    pdl_wait();
    constexpr int TILE = 32 * ILP;
    constexpr int kBytes = (int)Fp32cSmem<NW, ILP, TC>::bytes;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    float4 *s_red = reinterpret_cast<float4 *>(smem_raw) + Fp32cSmem<NW, ILP, TC>::red_offset;
    const int n = P.c.n, n_pad = P.c.n_pad;
    if constexpr (!CL) {
        const int S = P.split, r = (int)(blockIdx.x % (S * P.nsets)), set = r / S, rank = r % S;
        const int tile = blockIdx.x / (S * P.nsets), tid = threadIdx.x;
        fp32c_sweep<NW, ILP, TC, CULL>(StageView{P, P.buf[set]}, tile, rank, S, tid, [] { __syncthreads(); }, smem_raw);
        for (int e = tid; e < TILE; e += NW * 32)
            if (tile * TILE + e < n) {
                const float4 v = s_red[e];
                P.partial[(size_t)(2 * r) * n_pad + tile * TILE + e] = make_float2(v.x, v.z);
                P.partial[(size_t)(2 * r + 1) * n_pad + tile * TILE + e] = make_float2(v.y, v.w);
            }
    } else {
        static_assert(sizeof(EpilogueShared) * ILP <= Fp32cSmem<NW, ILP, TC>::tile, "epilogue over the j tile");
        const int S = (int)cg::this_cluster().num_blocks(), rank = (int)cg::this_cluster().block_rank();
        const int tile = blockIdx.x / S, set = threadIdx.x / (NW * 32), tid = threadIdx.x % (NW * 32);
        fp32c_sweep<NW, ILP, TC, CULL>(StageView{P, P.buf[set]}, tile, rank, S, tid, [&] { bar_sync(kBarSet + set, NW * 32); },
                                       smem_raw + set * kBytes);
        if (S > 1) cg::this_cluster().sync();
        else __syncthreads();
        if (rank == 0)
            tile_epilogue<ILP>(P, s_red, kBytes / 16, tile, S, reinterpret_cast<EpilogueShared *>(smem_raw));
        pass_step_advance(P);
        if (S > 1) cg::this_cluster().sync();  // the other blocks' sums stay readable until here
    }
}

// Sum over the j split's ranks, in rank order, of one axis's partials
// (s, c) of particle i at set e (each stands for s - c): the s exactly as an
// unevaluated float pair (TwoSum), the small c plainly, FP64 once -- FP64
// runs at ~1/64 of the FP32 rate here and an FP64 sum over the ranks
// dominated the finish.  Times C q_i (left out of the sweeps), in FP64.
__device__ __forceinline__ double finish_rank_sum(const StageParams &P, int i, int e, int axis) {
    TwoFloatSum sa;
    float ca = 0.0f;
    const float2 *p = P.partial + (size_t)(2 * e * P.split + axis) * P.c.n_pad + i;
    const size_t stride = 2 * (size_t)P.c.n_pad;
    int r = 0;
    for (; r + 16 <= P.split; r += 16) {  // 16 loads in flight, summed in rank order
        float2 v[16];
#pragma unroll
        for (int u = 0; u < 16; u++) v[u] = p[(size_t)(r + u) * stride];
#pragma unroll
        for (int u = 0; u < 16; u++) {
            sa.add(v[u].x);
            ca += v[u].y;
        }
    }
    for (; r + 8 <= P.split; r += 8) {  // 8 loads in flight, summed in rank order
        float2 v[8];
#pragma unroll
        for (int u = 0; u < 8; u++) v[u] = p[(size_t)(r + u) * stride];
#pragma unroll
        for (int u = 0; u < 8; u++) {
            sa.add(v[u].x);
            ca += v[u].y;
        }
    }
    for (; r < P.split; r++) {
        const float2 v = p[(size_t)r * stride];
        sa.add(v.x);
        ca += v.y;
    }
    // the two small corrections combined in FP32 (their rounding is ~2^-24
    // of ~2^-24 of the sum): two FP64 operations fewer per particle and axis
    return __dmul_rn(pair_scale(P, i), widen(sa.hi) + widen(sa.lo - ca));
}

// Completes a pass after a non-cluster pair launch: one block per
// 32-particle group, warp w < 2 nsets sums set w/2, axis w%2 over the ranks,
// then the first two warps run the epilogue.  ALL (forces outside
// kBasicForces): a block of 2 kTermParts warps, which first compute the
// position terms, a part of one set each (a chain of ~200 FP64 instructions on
// two warps otherwise; with one warp advancing both axes too, 4095 particles
// under every force took 17.2 us instead of 11.4).
template <bool ALL>
static __global__ void __launch_bounds__(ALL ? 64 * kTermParts : 128) stage_finish(const StageParams P) {
    pdl_wait();
    __shared__ EpilogueShared S;
    __shared__ double s_f[2][2][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int i = blockIdx.x * 32 + lane;
    if (i < P.c.n) {
        if (warp < 2) epilogue_prefetch(P, i, warp);  // the operands' round trip overlaps the partials'
        if (ALL && warp / kTermParts < P.nsets) {
            const int e = warp / kTermParts, b = P.buf[e];
            position_terms(S.terms[e][lane], warp % kTermParts, P.f, P.c.px[b][i], P.c.py[b][i], P.c.q[i],
                           (P.f.flags & kDriving) ? stage_time(P, e) : 0.0);
        }
        if (warp < 2 * P.nsets) s_f[warp >> 1][warp & 1][lane] = finish_rank_sum(P, i, warp >> 1, warp & 1);
    }
    __syncthreads();
    if (warp < 2)
        pass_epilogue<ALL>(P, EpilogueCloud{P.f, P.c.rc2_up, i < P.c.n, i >> 5}, i, warp, kBarEpilogue, s_f[0][warp][lane],
                           s_f[1][warp][lane], S);
    pass_step_advance(P);
}

// ---------------------------------------------------------------------------
// FP64 kernel: one 32-particle group of i per tile, S blocks per tile (a
// cluster), each with NW warps per position set; the j groups (CULL: those
// whose box is within reach of the tile's) are dealt one by one to the S*NW
// warps of a set, each of which filters its groups in FP32 and evaluates the
// hits in FP64 with full warps (dm_fp64.cuh).  The sums meet in the cluster's
// first block, which runs the epilogue.
//
// Bound by the FP64 pipe on dense clouds (20 FP64 instructions per pair that
// passed the filter and 2 to add it up, 64 cycles of a scheduler's FP64 unit per
// 32 pairs each), by latency on sparse ones.
// ---------------------------------------------------------------------------
template <int NW>
struct Group64Set {  // one position set's half of the block
    HitWarp<HitResult<2>> w[NW];
    double ix[32], iy[32];
    double2 acc[NW][32];
    double2 red[32];
    NearLists<NW, 1> near;
};
template <int NW>
struct Group64Smem {
    Group64Set<NW> set[2];
    double tab[kExp2Size];
    EpilogueShared epi;
};

template <int NW, bool CULL>
__global__ void __launch_bounds__(2 * NW * 32, 10 / NW) pair_group_fp64(const StageParams P) {
    pdl_wait();
    constexpr int NT = NW * 32;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    Group64Smem<NW> &sh = *reinterpret_cast<Group64Smem<NW> *>(smem_raw);
    cg::cluster_group cl = cg::this_cluster();
    const int S = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const int tile = blockIdx.x / S;
    const int set = threadIdx.x / NT, tid = threadIdx.x % NT, lane = tid & 31, warp = tid >> 5;
    Group64Set<NW> &sm = sh.set[set];
    const int n = P.c.n;
    const int i = tile * 32 + lane;
    const int b = P.buf[set];
    const double *__restrict__ px = P.c.px[b];
    const double *__restrict__ py = P.c.py[b];
    const double *__restrict__ qa = P.c.q;
    const float4 *__restrict__ pa = P.c.pa[b];
    const Yukawa64 K = P.y64;
    const bool coul = (P.f.flags & kShieldedCoulomb) != 0;
    // the warps that run the epilogue: see tile_epilogue
    const int npairs = blockDim.x >> 6, wib = threadIdx.x >> 5;
    const bool mine = rank == 0 && ((wib >> 1) + tile) % npairs == 0;
    double sum[2] = {0.0, 0.0};
    if (coul) {
        // every load of the prologue in flight at once
        float4 A = make_float4(0.0f, 0.0f, 0.0f, 0.0f), B = make_float4(0.0f, 0.0f, INFINITY, 0.0f);
        double xi = 0.0, yi = 0.0, tab[kExp2Size / NT];
        if (i < n) {
            A = pa[i];
            B = P.c.pb[b][i];
            xi = px[i];
            yi = py[i];
            if (mine) epilogue_prefetch(P, i, wib & 1);
        }
        if (set == 0)
#pragma unroll
            for (int k = 0; k < kExp2Size / NT; k++) tab[k] = g_exp2_table.v[k * NT + tid];
        if (warp == 0) {
            sm.ix[lane] = xi;
            sm.iy[lane] = yi;
        }
        if (set == 0)
#pragma unroll
            for (int k = 0; k < kExp2Size / NT; k++) sh.tab[k * NT + tid] = tab[k];
        const float px2 = 2.0f * A.x, py2 = 2.0f * A.y, nu = B.z;
        __syncthreads();
        HitWarp<HitResult<2>> &W = sm.w[warp];
        auto eval = [&](int il, int j) {
            const double dx = __dsub_rn(sm.ix[il], px[j]), dy = __dsub_rn(sm.iy[il], py[j]);
            const double w = pair_w64(dx, dy, qa[j], K, sh.tab);
            return HitResult<2>{__dmul_rn(w, dx), __dmul_rn(w, dy)};
        };
        int nk = 0, hits = 0;
        auto group = [&](int g) {
            const int j = 32 * g + lane;
            if (j < n) {
                prefetch_l1(px + j);
                prefetch_l1(py + j);
                prefetch_l1(qa + j);
            }
            hits += hit_filter(W, nk, g, tile, [&](int k) { return pa[k]; }, n, px2, py2, nu);
            if (++nk == kHitGroups || __reduce_add_sync(0xffffffffu, hits) >= 7 * 32) {
                __syncwarp();
                hit_flush(W, nk, sum, eval);
                nk = hits = 0;
            }
        };
        const int ngroups = (n + 31) >> 5;
        const int NS = NW * S, me = warp * S + rank;
        if constexpr (CULL) {
            const float4 tb = P.c.gbox[b][tile];
            int found = 0;
            for_near_groups(
                sm.near, P.c.gbox[b], P.c.gsuper[b], ngroups, 0, 1, tb, P.rc2_hi, tid,
                [&] { bar_sync(kBarSet + set, NT); }, [](int, const float4 &) { return 0; },
                [&](const int (&)[1], const int (&total)[1]) {
                    for (int e = (me + NS - found % NS) % NS; e < total[0]; e += NS) group(sm.near.list[e]);
                    found += total[0];
                });
            if (tid == 0 && rank == 0) atomicAdd(P.c.eval_pairs, 1024ull * (unsigned long long)found);
        } else {
            for (int g = me; g < ngroups; g += NS) group(g);
        }
        __syncwarp();
        hit_flush(W, nk, sum, eval);
    }
    sm.acc[warp][lane] = make_double2(sum[0], sum[1]);
    if (S > 1) {  // each block's sums, for the first block to read
        bar_sync(kBarSet + set, NT);
        if (warp == 0) {
            double2 t = sm.acc[0][lane];
#pragma unroll
            for (int w = 1; w < NW; w++) t = make_double2(__dadd_rn(t.x, sm.acc[w][lane].x), __dadd_rn(t.y, sm.acc[w][lane].y));
            sm.red[lane] = t;
        }
        cl.sync();
    } else {
        __syncthreads();
    }
    if (mine) {
        const int ax = wib & 1;
        const double cq = (i < n) ? __dmul_rn(P.coulomb, qa[i]) : 0.0;
        double f[2] = {0.0, 0.0};
        for (int e = 0; e < P.nsets; e++) {
            double t = 0.0;
            const int terms = (S > 1) ? S : NW;
            for (int k = 0; k < terms; k++) {
                const double2 v = (S > 1) ? *cl.map_shared_rank(&sh.set[e].red[lane], k) : sh.set[e].acc[k][lane];
                t = __dadd_rn(t, ax ? v.y : v.x);
            }
            f[e] = __dmul_rn(cq, t);
        }
        pass_epilogue(P, EpilogueCloud{P.f, P.c.rc2_up, i < n, tile}, i, ax, kBarEpilogue, f[0], f[1], sh.epi);
    }
    pass_step_advance(P);
    if (S > 1) cl.sync();  // the other blocks' sums stay readable until here
}

}  // namespace dm
