// dm_fp64.cuh -- FP64 pair arithmetic for a GPU whose FP64 units run at 1/64
// of its FP32 rate, and the culled FP64 pair + stage kernel built on it.
//
// An FP64 instruction of a warp occupies an SM's FP64 pipe for 16 cycles
// however many of its lanes are active; in that time the SM issues 64 other
// instructions.  So everything but the pair terms themselves is kept off the
// FP64 pipe, and the pair terms always run with full warps:
//   * which pairs are near the cutoff is found in FP32 (the conservative
//     filter of filter_threshold), a 32 x 32 bit mask per pair of groups;
//   * a warp collects the masks of several j groups, lays the hits out as
//     one dense list (codes in shared memory, ordered by i), evaluates 32
//     list entries per round, whatever i and j they belong to, and every
//     lane then adds up its own particle's entries in list order
//     (deterministic, no atomics);
//   * 1/r, r and e^{-kappa r} take 9 FP64 instructions (yukawa64) instead
//     of a square root, a division and an exponential of the math library
//     (~70); conversions between the two precisions are integer operations.
#pragma once

#include <cooperative_groups.h>

#include <cmath>
#include <cstring>

#include "dm_device.cuh"

namespace dm {
namespace cg = cooperative_groups;

// 2^(k/512), k = 0..511, correctly rounded: the Taylor series of
// exp(k ln2/512) in unevaluated double pairs (~100 bits), at compile time.
constexpr int kExp2Bits = 9;
constexpr int kExp2Size = 1 << kExp2Bits;
struct Exp2Table {
    double v[kExp2Size];
};
struct DD {
    double hi, lo;
};
constexpr DD dd_add(DD a, DD b) {  // Knuth's TwoSum, low parts added plainly
    const double s = a.hi + b.hi, t = s - a.hi;
    const double e = ((a.hi - (s - t)) + (b.hi - t)) + (a.lo + b.lo);
    const double h = s + e;
    return {h, e - (h - s)};
}
constexpr DD dd_mul(DD a, DD b) {  // Dekker's product
    const double c = 134217729.0;  // 2^27 + 1
    const double ca = c * a.hi, cb = c * b.hi;
    const double ah = ca - (ca - a.hi), al = a.hi - ah;
    const double bh = cb - (cb - b.hi), bl = b.hi - bh;
    const double p = a.hi * b.hi;
    const double e = (((ah * bh - p) + ah * bl + al * bh) + al * bl) + (a.hi * b.lo + a.lo * b.hi);
    const double h = p + e;
    return {h, e - (h - p)};
}
constexpr Exp2Table make_exp2_table() {
    // ln 2 as an unevaluated pair
    const DD ln2{0.6931471805599453, 2.3190468138462996e-17};
    // Horner's scheme in x/j, 1/j as a pair by one Newton correction of the
    // double quotient
    Exp2Table t{};
    for (int k = 0; k < kExp2Size; k++) {
        const DD x = dd_mul(ln2, DD{(double)k / kExp2Size, 0.0});
        DD s{1.0, 0.0};
        for (int j = 30; j >= 1; j--) {
            const double inv = 1.0 / j;
            const DD one = dd_mul(DD{inv, 0.0}, DD{(double)j, 0.0});
            const DD rec{inv, -((one.hi - 1.0) + one.lo) * inv};
            s = dd_add(DD{1.0, 0.0}, dd_mul(dd_mul(x, rec), s));
        }
        t.v[k] = s.hi;
    }
    return t;
}
static __device__ const Exp2Table g_exp2_table = make_exp2_table();

constexpr double kExp2C1 = 0.0013538030870311431;  // ln2/512

inline Yukawa64 make_yukawa64(double kappa, double rc2) {
    Yukawa64 K;
    const double l_hi = 738.6598609351493, l_lo = 1.0421900155356689e-14;  // 512 log2(e)
    K.kappa = kappa;
    K.k_hi = -(kappa * l_hi);
    K.k_lo = (float)(-(std::fma(kappa, l_hi, K.k_hi) + kappa * l_lo) * kExp2C1);
    K.k_f = (float)K.k_hi;
    uint64_t w;
    std::memcpy(&w, &rc2, sizeof w);
    K.rc2_word = (uint32_t)(w >> 32);
    return K;
}

// Values of one pair at squared distance r2: y = 1/r, ex = e^{-kappa r} and
// kappa r (formed only by callers that use it: r y kappa).
struct Yukawa64At {
    double y, r, ex;
};

// r2 in [2^-100, 2^100): 5 FP64 instructions for 1/r and r (a third-order
// step from the FP32 reciprocal square root, 2^-22; e^3 < 2^-63), 4 for the
// exponential (table of 512, degree-4 polynomial, |remainder| < 2e-18).
// -kappa r enters as k r with k a pair, rounded once after the integer part
// is taken off, so the exponential's error does not grow with kappa r.
//
// Where a term is so small that FP32 gives it to beyond the result's last
// bit, it is evaluated there: the step's second order (3/8 e^2 < 2^-44 of 1/r),
// k's low part (2^-50 of the exponential), and the polynomial's third and
// fourth degree (f c3 + f^2 c4, 2^-11 of c2, added to c2's bits as an
// integer).  The same errors against long double as all 13 operations in FP64
// (1/r 1.4e-16, r 1.2e-16, exponential 1.0e-15 at most for kappa r < 10, kappa
// 1 .. 3e7).  With 13: a pair 24 FP64 instructions instead of 20, a 6-cloud
// gradient 19.6 -> 17.2 ms, 100 steps of 512 grains 3.06 -> 2.83 ms.
__device__ __forceinline__ Yukawa64At yukawa64(double r2, const Yukawa64 &K, const double *tab) {
    const uint32_t lo = (uint32_t)__double2loint(r2), hi = (uint32_t)__double2hiint(r2);
    const float rf = __uint_as_float(__funnelshift_l(lo, hi - 0x38000000u, 3));  // truncated to FP32
    float yf;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(yf) : "f"(rf));
    const uint32_t yb = __float_as_uint(yf);
    const double y0 = __hiloint2double((int)((yb >> 3) + 0x38000000u), (int)(yb << 29));  // exact
    const double t = __dmul_rn(r2, y0);
    const double e = fma(-t, y0, 1.0);
    const float ef = narrow(e), r_f = rf * yf;
    const double h = fma(e, 0.5, widen_normal(0.375f * ef * ef));
    Yukawa64At A;
    A.y = fma(y0, h, y0);
    A.r = fma(t, h, t);
    // n = the integer nearest k r (any integer within ~0.51 of it will do)
    const float nf = rintf(r_f * K.k_f);
    const int n = (int)nf;  // <= 0
    const uint32_t nb = __float_as_uint(nf) & 0x7FFFFFFFu;
    // -n as a double (n = 0 gives 2^-127: no matter)
    const double nd = __hiloint2double((int)((nb >> 3) + 0x38000000u), (int)(nb << 29));
    const double f = fma(A.r, K.k_hi, nd);
    // c_m = (ln2/512)^m / m!; c2 + (f c3 + f^2 c4) in c2's binade, whose last
    // place is 2^-73: the sum in units of 2^-62, |f| <= 0.53
    constexpr float kUnit = 4611686018427387904.0f;  // 2^62
    constexpr long long kC2 = 0x3EAEBFBDFF82C58FLL;  // 9.163913992275266e-07
    const float ff = narrow(f);
    const int c34 = __float2int_rn(ff * fmaf(ff, 1.399621994296973e-13f * kUnit, 4.135378350676714e-10f * kUnit));
    const double q = __longlong_as_double(kC2 + ((long long)c34 << 11));
    const double p = fma(f, fma(f, q, kExp2C1), widen_normal(r_f * K.k_lo));
    const double T0 = tab[n & (kExp2Size - 1)];
    const double T = __hiloint2double(__double2hiint(T0) + ((n >> kExp2Bits) << 20), __double2loint(T0));
    A.ex = fma(T, p, T);
    return A;
}

// Whether a pair is inside the cutoff, bit for bit as the reference decides:
// by r2's high word away from the cutoff, else by its own operations.
__device__ __forceinline__ bool in_cutoff64(double dx, double dy, double r2, const Yukawa64 &K) {
    const uint32_t w = (uint32_t)__double2hiint(r2);
    if (w + 1u < K.rc2_word) return true;  // r2 < r_c^2 (1 - 2^-21): rounding cannot matter
    if (w > K.rc2_word + 1u) return false;
    double r, a;
    return ref_in_cutoff(dx, dy, K.kappa, r, a);
}

// r2 outside yukawa64's range (no cloud in SI units gets here; NaN does)
__device__ __forceinline__ bool yukawa64_odd(double r2) {
    return (uint32_t)__double2hiint(r2) - (923u << 20) >= (200u << 20);
}
static __device__ __noinline__ Yukawa64At yukawa64_general(double r2, double kappa) {
    Yukawa64At A;
    A.r = sqrt(r2);
    A.y = 1.0 / A.r;
    A.ex = exp(-kappa * A.r);
    return A;
}

// w of one pair, the force on i from j being C q_i w (dx, dy):
// w = q_j (1 + kappa r) e^{-kappa r} / r^3 = q_j e^{-kappa r} y^2 (y + kappa)
// (ShieldedCoulombForce.cpp:144-157); 0 outside the cutoff.
__device__ __forceinline__ double pair_w64(double dx, double dy, double qj, const Yukawa64 &K, const double *tab) {
    const double r2 = fma(dx, dx, __dmul_rn(dy, dy));
    const bool in = in_cutoff64(dx, dy, r2, K);
    Yukawa64At A;
    if (yukawa64_odd(r2)) A = yukawa64_general(r2, K.kappa);
    else A = yukawa64(r2, K, tab);
    const double w = __dmul_rn(__dmul_rn(qj, A.ex), __dmul_rn(__dmul_rn(A.y, A.y), __dadd_rn(A.y, K.kappa)));
    return in ? w : 0.0;
}

// ---------------------------------------------------------------------------
// The hit list of one warp: masks of up to kHitGroups j groups against the
// warp's 32 i particles, evaluated in windows of up to kHitPerLane hits of
// every i.
// ---------------------------------------------------------------------------
constexpr int kHitGroups = 8;
constexpr int kHitPerLane = 8;

template <int NS>
struct HitResult {
    double v[NS];
};

template <class Result>
struct alignas(16) HitWarp {
    Result res[kHitPerLane * 32];     // the entries' results
    float fx[32], fy[32], fb[32];     // the j group being filtered: xh, yh, -|p|^2
    uint32_t mask[kHitGroups][32];    // bit jl of mask[k][il]: pair (il, group k's jl)
    int group[kHitGroups];            // the j groups
    uint16_t code[kHitPerLane * 32];  // (k << 10) | (jl << 5) | il
};

// Filters j group g (FP32 position of j: load(j) = (xh, yh, |p|^2, -); n particles) against this lane's i
// (px2 = 2 xh_i, py2 = 2 yh_i, nu = -bound_i; nu = INFINITY: no particle) and
// stores the lane's mask as entry k.  A pair is out if bound_i - |p_j|^2 + 2
// p_i.p_j is negative (two j per packed instruction, 3 instructions per pair);
// NaN passes: such a pair is decided later.  Returns the lane's number of hits.
template <class Result, class Load>
__device__ __forceinline__ int hit_filter(HitWarp<Result> &W, int k, int g, int self, Load load, int n, float px2,
                                          float py2, float nu) {
    const int lane = threadIdx.x & 31;
    const int j = 32 * g + lane;
    const float4 A = (j < n) ? load(j) : make_float4(0.0f, 0.0f, INFINITY, 0.0f);
    __syncwarp();
    W.fx[lane] = A.x;
    W.fy[lane] = A.y;
    W.fb[lane] = -A.z;
    if (lane == 0) W.group[k] = g;
    __syncwarp();
    const float2 p2 = make_float2(px2, px2), q2 = make_float2(py2, py2), nb = make_float2(-nu, -nu);
    uint32_t m = 0u;
#pragma unroll
    for (int c = 7; c >= 0; c--) {
        const float4 X = reinterpret_cast<const float4 *>(W.fx)[c], Y = reinterpret_cast<const float4 *>(W.fy)[c],
                     B = reinterpret_cast<const float4 *>(W.fb)[c];
        const float2 t01 = __ffma2_rn(p2, make_float2(X.x, X.y),
                                      __ffma2_rn(q2, make_float2(Y.x, Y.y), __fadd2_rn(make_float2(B.x, B.y), nb)));
        const float2 t23 = __ffma2_rn(p2, make_float2(X.z, X.w),
                                      __ffma2_rn(q2, make_float2(Y.z, Y.w), __fadd2_rn(make_float2(B.z, B.w), nb)));
        m = __funnelshift_l(__float_as_uint(t23.y), m, 1);
        m = __funnelshift_l(__float_as_uint(t23.x), m, 1);
        m = __funnelshift_l(__float_as_uint(t01.y), m, 1);
        m = __funnelshift_l(__float_as_uint(t01.x), m, 1);
    }
    m = ~m;
    if (nu == INFINITY) m = 0u;
    if (g == self) m &= ~(1u << lane);  // j == i
    const int left = n - 32 * g;
    if (left < 32) m &= (1u << left) - 1u;
    W.mask[k][lane] = m;
    return __popc(m);
}

// Lays every hit of the first `ng` masks out in windows of up to kHitPerLane
// hits of every i: work(total) runs on the window's entries (code[0 ..
// total-1], ordered by i), then collect(off, c) on every lane with the range of
// its own i's entries, in the order (k, jl).
template <class Result, class Work, class Collect>
__device__ __forceinline__ void hit_windows(HitWarp<Result> &W, int ng, Work work, Collect collect) {
    const int lane = threadIdx.x & 31;
    int k = 0;
    uint32_t m = (ng > 0) ? W.mask[0][lane] : 0u;
    for (;;) {
        int left = __popc(m);
        for (int kk = k + 1; kk < ng && left < kHitPerLane; kk++) left += __popc(W.mask[kk][lane]);
        const int c = min(left, kHitPerLane);
        int off = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, off, o);
            if (lane >= o) off += v;
        }
        const int total = __shfl_sync(0xffffffffu, off, 31);
        if (total == 0) break;
        off -= c;
        for (int t = 0; t < c; t++) {
            while (m == 0u) m = W.mask[++k][lane];
            const int u = __ffs(m) - 1;
            m &= m - 1u;
            W.code[off + t] = (uint16_t)((k << 10) | (u << 5) | lane);
        }
        __syncwarp();
        work(total);
        __syncwarp();
        collect(off, c);
        __syncwarp();
    }
}

// FP64: eval(il, j) gives an entry's result, summed per i into sum[NS].
template <int NS, class Eval>
__device__ __forceinline__ void hit_flush(HitWarp<HitResult<NS>> &W, int ng, double (&sum)[NS], Eval eval) {
    hit_windows(
        W, ng,
        [&](int total) {
            for (int t = threadIdx.x & 31; t < total; t += 32) {
                const int code = W.code[t];
                W.res[t] = eval(code & 31, 32 * W.group[code >> 10] + ((code >> 5) & 31));
            }
        },
        [&](int off, int c) {
            for (int t = 0; t < c; t++) {
#pragma unroll
                for (int e = 0; e < NS; e++) sum[e] = __dadd_rn(sum[e], W.res[off + t].v[e]);
            }
        });
}

// Calls eval(il, 32 k + jl) for every bit of the warp's masks mask[k][il],
// k < ng, 32 hits at a time (windows of up to kHitSumPerLane hits of every
// i); `code` is the warp's scratch.
constexpr int kHitSumPerLane = 16;
template <class Eval>
__device__ __forceinline__ void hit_sum(const uint32_t (*mask)[32], int ng, uint16_t *code, Eval eval) {
    const int lane = threadIdx.x & 31;
    int k = 0;
    uint32_t m = (ng > 0) ? mask[0][lane] : 0u;
    for (;;) {
        int left = __popc(m);
        for (int kk = k + 1; kk < ng && left < kHitSumPerLane; kk++) left += __popc(mask[kk][lane]);
        const int c = min(left, kHitSumPerLane);
        int off = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, off, o);
            if (lane >= o) off += v;
        }
        const int total = __shfl_sync(0xffffffffu, off, 31);
        if (total == 0) break;
        off -= c;
        for (int t = 0; t < c; t++) {
            while (m == 0u) m = mask[++k][lane];
            const int u = __ffs(m) - 1;
            m &= m - 1u;
            code[off + t] = (uint16_t)((lane << 8) | (32 * k + u));
        }
        __syncwarp();
        for (int t = lane; t < total; t += 32) eval(code[t] >> 8, code[t] & 255);
        __syncwarp();
    }
}

// FP32 candidate test, conservative for the FP64 cutoff decision.  With
// xf = fl32(x) (|xf - x| <= 2^-24 |x|) and dxf = fl32(xf_i - xf_j), the error of
// dxf is at most 2^-24 (|x_i| + |x_j|) + 2^-24 |dxf| <= e = 2^-22 (A_i + A_t),
// where A_i = max(|x_i|, |y_i|) and A_t bounds |x_j|, |y_j| over the j tile; the
// error vector of (dxf, dyf) is shorter than 2e.  So every pair with true
// r < r_c has fl32(dxf^2 + dyf^2) < (r_c + 2e)^2 (1 + 2^-20) -- the last factor
// covers the three FP32 roundings of the square sum and of r_c itself.  The
// exact decision is then the reference's FP64 test (ref_in_cutoff).
__device__ __forceinline__ float candidate_bound(double rc, float ai, float at) {
    const float e = 2.384185791015625e-7f * (ai + at);  // 2^-22
    const float r = __fadd_ru(__double2float_ru(rc), 2.0f * e);
    return __fmul_ru(__fmul_ru(r, r), 1.0000009536743164f);  // 1 + 2^-20
}

}  // namespace dm
