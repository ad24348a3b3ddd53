// dm_device.cuh -- device-side data layout and per-particle arithmetic of the
// DEMON hot path on sm_103a.
//
// A step runs in passes of two force evaluations each.  The position an RK
// stage evaluates the pair force at depends only on the velocity before the
// previous stage's force (x2 = x + dt v/2 is known with the state, x3 = x + dt
// v2/2 needs F1, x4 = x + dt v3 needs F2), so RK4's four pair sums are two
// launches of two independent position sets: pass 0 evaluates F at x1 and x2
// and its epilogue forms v2, v3, x3, x4; pass 1 evaluates F at x3 and x4 and
// ends the step, forming the next step's x2 as well.  RK2 (stages x and x2) is
// one pass.  The arithmetic of each particle is the reference's, operation for
// operation.
//
// Layout in HBM (one cloud, n particles padded to n_pad, a multiple of 64):
//   base state       x, y, vx, vy, q, m                      FP64 [n_pad]
//   increments       k1[2], k2[2] (dt F/m of stages 1, 2; x and y), 1/m  FP64 [n_pad]
//   position sets    b = 0: x1 = the state, 1: x2, 2: x3, 3: x4; per set
//                      px[b], py[b]  FP64 (CacheOperator's xCache/yCache);
//                                    px[0], py[0] are x, y themselves
//                      pa[b] = (xh, yh, xh^2+yh^2, (float)q)  float4
//                      pb[b] = (xl, yl, -threshold, 0)        float4
//                    (threshold = the FP32 pair filter's bound, see
//                    filter_threshold; computed once per particle here
//                    instead of in every CTA that reads the particle)
//                    with x = xh + xl exactly to 48 bits (two-float form).
//   padding          particles n..n_pad-1 sit at 1e18 m with q = 0, so the
//                    cutoff test never selects them.
#pragma once

#include <cfloat>
#include <cmath>
#include <cstdint>
#include <utility>
#include <cuda_runtime.h>

namespace dm {

// ForceFlag bits (Force.h:75-91)
constexpr long long kConfinement = 1;
constexpr long long kDrag = 2;
constexpr long long kShieldedCoulomb = 4;
constexpr long long kGravitational = 8;
constexpr long long kThermal = 16;
constexpr long long kThermalLocalized = 32;
constexpr long long kDriving = 64;
constexpr long long kRotational = 128;
constexpr long long kTimeVaryingDrag = 256;
constexpr long long kTimeVaryingThermal = 512;
constexpr long long kMagnetic = 1024;
constexpr long long kConfinementVoid = 2048;
constexpr long long kElectric = 4096;
constexpr long long kRectConfinement = 8192;
constexpr long long kVertElectric = 16384;
constexpr long long kAllForces = 32767;
// forces that read the force time
constexpr long long kTimeForces = kDriving | kTimeVaryingDrag | kTimeVaryingThermal;
// Forces whose x and y components are independent (the fast epilogue path)
constexpr long long kBasicForces = kConfinement | kDrag | kRectConfinement | kShieldedCoulomb | kThermal;

constexpr float kPadPosition = 1.0e18f;

struct ForceParams {  // same layout as dm_force_params
    long long flags;
    double shielding, confine, confine_x, confine_y, gamma, heat;
    int thermal_mode, reserved;
    unsigned long long seed;
    double void_decay, drive_const, drive_amplitude, drive_shift, magnetic, rot_rmin, rot_rmax, rot_const;
    double heat_in, heat_out, heat_radius, drag_scale, drag_offset, heat_scale, heat_offset;
    double electric, electric_radius, gravity, vert_electric, vert_decay;
};

struct CloudDev {
    int n, n_pad;
    double *x, *y, *vx, *vy, *q, *m;
    double *k1[2], *k2[2];
    double *invm;                  // 1/m, kept with m (a reciprocal is 9 FP64 instructions)
    double *px[4], *py[4];
    float4 *pa[4], *pb[4];
    float4 *gbox[4];               // [n_pad/32] FP32 box (x0, y0, x1, y1) of each 32-particle group
    float4 *gsuper[4];             // box of every 32 groups (large clouds; else nullptr)
    unsigned long long *eval_pairs;  // ordered pairs the culling kernels swept (cumulative)
    unsigned long long *step_ctr;  // [3], see pass_step_index()
    double *time;                  // [3] force time slots, see stage_time()
    int *err;                      // device error flags
    double rc2;                    // (10/kappa)^2 of the current force parameters
    float rc2_up;                  // the same rounded up to FP32
    double coulomb;                // 1/(4 pi eps0)
    int *orig;                     // caller's index of internal slot s (Morton order)
};

// An RK2 step's results (sets 2 and 3) become the state and its midpoint (host).
inline void swap_sets(CloudDev &c) {
    for (int b = 0; b < 2; b++) {
        std::swap(c.px[b], c.px[b + 2]);
        std::swap(c.py[b], c.py[b + 2]);
        std::swap(c.pa[b], c.pa[b + 2]);
        std::swap(c.pb[b], c.pb[b + 2]);
        std::swap(c.gbox[b], c.gbox[b + 2]);
        std::swap(c.gsuper[b], c.gsuper[b + 2]);
    }
    c.x = c.px[0];
    c.y = c.py[0];
}

// Host-side check of a force parameter set, shared by every entry point that
// takes one: DM_OK (0), or a status with *why set to a static message.
// Flags must be among the fifteen ForceFlag bits (status 6, unsupported);
// with ShieldedCoulomb on, kappa must be positive and finite (the cutoff is
// kappa*r < 10) and thermal_mode must be 0 or 1 (status 1, bad argument).
inline int check_force_params(const ForceParams &p, const char **why) {
    if (p.flags & ~kAllForces) {
        *why = "unknown force flags";
        return 6;
    }
    if ((p.flags & kShieldedCoulomb) && !(p.shielding > 0.0 && p.shielding <= DBL_MAX)) {
        *why = "shielding must be positive and finite";
        return 1;
    }
    if (p.thermal_mode != 0 && p.thermal_mode != 1) {
        *why = "thermal_mode must be 0 or 1";
        return 1;
    }
    return 0;
}

enum StageMode : int { kModeStep = 0, kModeForceOnly = 1 };

// Constants of the FP64 pair terms of one cloud (make_yukawa64).
struct Yukawa64 {
    double kappa;
    double k_hi;        // -kappa 512 log2(e)
    float k_f;          // the same in FP32
    float k_lo;         // what k_hi lacks, times ln2/512
    uint32_t rc2_word;  // high word of r_c^2: r^2 with a smaller one is inside the cutoff
};

// Everything a stage kernel needs, passed by value.
struct StageParams {
    CloudDev c;
    ForceParams f;
    int pass;             // 0 (stages 1, 2), 1 (stages 3, 4)
    int order;            // 4: Runge_Kutta4; 2: Runge_Kutta2 (the midpoint method)
    int mode;             // StageMode
    int nsets;            // position sets evaluated: 2 (steps), 1 (force-only; 2 when the autotuner times)
    int buf[2];           // the sets' buffers (force-only: 0 = the state, or the autotuner's copy)
    int slot;             // step counter / force time slot holding the current values (0 or 1)
    int therm_stage;      // force-only: substep index of the thermal kicks (any of 1..4)
    double dt;            // fixed dt (used when dt_dev == nullptr)
    const double *dt_dev; // adaptive dt computed on the device
    double coulomb;       // 1/(4 pi eps0)
    double *fx_out, *fy_out;  // kModeForceOnly outputs
    // pair-kernel constants
    double rc2;           // (10/kappa)^2
    float rc2_lo, rc2_hi; // FP32 certain-in / certain-out bounds on r^2
    float kappa_f;
    float nkl2e;          // -kappa*log2(e): e^{-kappa r} = 2^{nkl2e r}
    Yukawa64 y64;
    // FP32C sweep: 8 filtered chunks whose j pass the filter for at least
    // this many of every 128 (lane, j) pairs of a slot are evaluated directly
    // (all lanes, cutoff by a select) instead of through per-lane hit bits
    int direct_min;
    // culling: a near group whose farthest separation from the tile is
    // within sqrt(near_direct_f2) r_c skips the filter (every chunk
    // evaluated directly); 0: no such class
    float near_direct_f2;
    // j split without clusters: rank r of (tile t, set e) is block (t*nsets +
    // e)*split + r and writes its partial sums (s, c) of particle i to the
    // float2 planes partial[(2(e*split + r) + axis)*n_pad + i]; stage_finish
    // sums them
    int split;
    float2 *partial;
};

// FP32 to FP64 by integer operations (a conversion holds the FP64 unit).
// Zero, denormal and non-finite values take the conversion.
__device__ __forceinline__ double widen(float v) {
    const uint32_t b = __float_as_uint(v), e = (b >> 23) & 0xFFu;
    if (e - 1u >= 254u) return (double)v;
    return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7FFFFFFFu) >> 3) + 0x38000000u)), (int)(b << 29));
}

// A double rounded toward zero to FP32, by integer operations; 0 below 2^-126.
// |v| < 2^128.
__device__ __forceinline__ float narrow(double v) {
    const uint32_t h = (uint32_t)__double2hiint(v), m = h & 0x7FFFFFFFu;
    const uint32_t b = __funnelshift_l((uint32_t)__double2loint(v), m - 0x38000000u, 3);
    return __uint_as_float((h & 0x80000000u) | (m < 0x38100000u ? 0u : b));
}
// widen for a normal number or one too small to matter (zero gives 2^-127).
__device__ __forceinline__ double widen_normal(float v) {
    const uint32_t b = __float_as_uint(v);
    return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7FFFFFFFu) >> 3) + 0x38000000u)), (int)(b << 29));
}

// ---------------------------------------------------------------------------
// Counter-based RNG: Philox4x32-10 (Salmon, Moraes, Dror, Shaw, SC'11).
// ---------------------------------------------------------------------------
__device__ __forceinline__ void philox4x32_10(uint32_t c[4], uint32_t k0, uint32_t k1) {
    const uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u;
    const uint32_t W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
#pragma unroll
    for (int r = 0; r < 10; r++) {
        const uint32_t hi0 = __umulhi(M0, c[0]), lo0 = M0 * c[0];
        const uint32_t hi1 = __umulhi(M1, c[2]), lo1 = M1 * c[2];
        const uint32_t n0 = hi1 ^ c[1] ^ k0, n2 = hi0 ^ c[3] ^ k1;
        c[0] = n0; c[1] = lo1; c[2] = n2; c[3] = lo0;
        k0 += W0; k1 += W1;
    }
}

// Thermal kick arithmetic: FP32 Box-Muller built only from correctly rounded
// IEEE single operations (add, mul, fma, div, sqrt) in a fixed order, so the
// CPU oracle reproduces it bit for bit (oracle/demon_oracle.c).  The kick is
// noise of relative size ~1e-5 of the forces it is added to; FP32 (rather
// than FP64, which runs at 1/64 of the FP32 rate on this GPU) loses nothing.
//
// u in (0, 1): 24 random bits, (k + 0.5) * 2^-24.
__device__ __forceinline__ float u24(uint32_t w) {
    return __fmul_rn(__fadd_rn((float)(w >> 8), 0.5f), 5.9604644775390625e-8f);
}

// ln(u), u in (0, 1]: u = 2^e m with m in [sqrt(1/2), sqrt(2)),
// ln m = 2 atanh(s), s = (m-1)/(m+1), atanh by its odd series to s^9
// (|s| < 0.1716: truncation < 2e-9).
__device__ __forceinline__ float thermal_log(float u) {
    const uint32_t bits = __float_as_uint(u);
    int e = (int)(bits >> 23) - 127;
    float m = __uint_as_float((bits & 0x007FFFFFu) | 0x3F800000u);
    if (m > 1.41421356f) {
        m = __fmul_rn(m, 0.5f);
        e += 1;
    }
    const float s = __fdiv_rn(__fsub_rn(m, 1.0f), __fadd_rn(m, 1.0f));
    const float s2 = __fmul_rn(s, s);
    float p = __fmaf_rn(s2, 0.111111111f, 0.142857143f);
    p = __fmaf_rn(s2, p, 0.2f);
    p = __fmaf_rn(s2, p, 0.333333333f);
    p = __fmaf_rn(s2, p, 1.0f);
    const float lnm = __fmul_rn(__fmul_rn(2.0f, s), p);
    return __fmaf_rn((float)e, 0.693147181f, lnm);
}

// sin and cos of 2 pi u, u in [0, 1): quadrant q = floor(4u), a = (4u - q) pi/2
// in [0, pi/2), Taylor polynomials to a^13 (sin) and a^14 (cos), truncation
// < 7e-10, then the exact quadrant rotation.
__device__ __forceinline__ void thermal_sincos(float u, float &sn, float &cs) {
    const float r = __fmul_rn(u, 4.0f);
    const float qf = floorf(r);
    const int q = (int)qf;
    const float a = __fmul_rn(__fsub_rn(r, qf), 1.57079633f);
    const float a2 = __fmul_rn(a, a);
    float ps = __fmaf_rn(a2, 1.60590438e-10f, -2.50521084e-8f);
    ps = __fmaf_rn(a2, ps, 2.75573192e-6f);
    ps = __fmaf_rn(a2, ps, -1.98412698e-4f);
    ps = __fmaf_rn(a2, ps, 8.33333333e-3f);
    ps = __fmaf_rn(a2, ps, -1.66666667e-1f);
    ps = __fmaf_rn(a2, ps, 1.0f);
    const float sa = __fmul_rn(a, ps);
    float pc = __fmaf_rn(a2, -1.14707456e-11f, 2.08767570e-9f);
    pc = __fmaf_rn(a2, pc, -2.75573192e-7f);
    pc = __fmaf_rn(a2, pc, 2.48015873e-5f);
    pc = __fmaf_rn(a2, pc, -1.38888889e-3f);
    pc = __fmaf_rn(a2, pc, 4.16666667e-2f);
    pc = __fmaf_rn(a2, pc, -0.5f);
    const float ca = __fmaf_rn(a2, pc, 1.0f);
    switch (q & 3) {
        case 0: sn = sa; cs = ca; break;
        case 1: sn = ca; cs = -sa; break;
        case 2: sn = -sa; cs = -ca; break;
        default: sn = -ca; cs = sa; break;
    }
}

// Counter-based kick of scale `heat` for particle i: counter (i, step lo,
// step hi, stream).  Mode 0 is the reference's form heatVal*U*(cos t, sin t),
// t ~ U(0, 2pi) (ThermalForce.cpp:118-140) with counter-based uniforms; mode
// 1 is a Gaussian of standard deviation `heat` per axis (Box-Muller).
// Streams: stage for ThermalForce, stage + 16 for ThermalForceLocalized,
// stage + 32 for TimeVaryingThermalForce.
__device__ __forceinline__ void thermal_draw(const ForceParams &f, uint32_t i,
                                             unsigned long long step, int stream, double heat,
                                             double &tx, double &ty) {
    uint32_t c[4] = {i, (uint32_t)step, (uint32_t)(step >> 32), (uint32_t)stream};
    philox4x32_10(c, (uint32_t)f.seed, (uint32_t)(f.seed >> 32));
    const float u1 = u24(c[0]);
    const float u2 = u24(c[1]);
    float sn, cs;
    thermal_sincos(u2, sn, cs);
    float amp;
    if (f.thermal_mode == 0) amp = u1;
    else amp = __fsqrt_rn(__fmul_rn(-2.0f, thermal_log(u1)));
    tx = __dmul_rn(heat, widen(__fmul_rn(amp, cs)));
    ty = __dmul_rn(heat, widen(__fmul_rn(amp, sn)));
}

__device__ __forceinline__ void thermal_kick(const ForceParams &f, uint32_t i,
                                             unsigned long long step, int stage,
                                             double &tx, double &ty) {
    thermal_draw(f, i, step, stage, f.heat, tx, ty);
}

// RNG step index of the running pass.  RK4: pass 0 reads slot P.slot and
// copies it to slot 2; pass 1 reads slot 2 and advances slot P.slot.  RK2's
// one pass reads slot P.slot and writes the other one, which the host makes
// current.  Each slot is written only in a launch that never reads it, so no
// launch races itself.
__device__ __forceinline__ int pass_slot(const StageParams &P) {
    return (P.mode != kModeForceOnly && P.pass == 1) ? 2 : P.slot;
}
__device__ __forceinline__ unsigned long long pass_step_index(const StageParams &P) {
    return P.c.step_ctr[pass_slot(P)];
}
__device__ __forceinline__ double stage_dt(const StageParams &P) {
    return P.dt_dev ? *P.dt_dev : P.dt;
}
// Force time of set e of the running pass: t, t + dt/2.0, t + dt/2.0, t + dt
// for RK4 stages 1-4 (Runge_Kutta4.cpp:30-88), t, t + dt/2.0 for RK2 stages
// 1-2 (Runge_Kutta2.cpp:28-50), t the time at the start of the step, kept as
// the step counter is; the last pass leaves t + dt (currentTime += dt,
// Runge_Kutta4.cpp:135, Runge_Kutta2.cpp:76).  Force-only launches use the
// current time.
__device__ __forceinline__ double stage_time(const StageParams &P, int e) {
    const double t = P.c.time[pass_slot(P)];
    if (P.mode == kModeForceOnly || (P.pass == 0 && e == 0)) return t;
    const double dt = stage_dt(P);
    return (P.pass == 1 && e == 1) ? __dadd_rn(t, dt) : __dadd_rn(t, __ddiv_rn(dt, 2.0));
}
// Substep index of set e's thermal kicks.
__device__ __forceinline__ int thermal_stage(const StageParams &P, int e) {
    return (P.mode == kModeForceOnly) ? P.therm_stage : 2 * P.pass + e + 1;
}
__device__ __forceinline__ void pass_step_advance(const StageParams &P) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    if (P.mode == kModeForceOnly) return;
    if (P.order == 4 && P.pass == 0) {
        P.c.step_ctr[2] = P.c.step_ctr[P.slot];
        P.c.time[2] = P.c.time[P.slot];
    } else {
        const int from = pass_slot(P), to = (P.order == 2) ? P.slot ^ 1 : P.slot;
        P.c.step_ctr[to] = P.c.step_ctr[from] + 1ull;
        P.c.time[to] = __dadd_rn(P.c.time[from], stage_dt(P));
    }
}

// Two-float split of a position: x = hi + lo, hi = x rounded to FP32, lo the
// remainder rounded to FP32.  Integer operations on x's bits (the remainder of
// a mantissa rounded to 24 bits is an integer of at most 29): the same values
// as two conversions, a conversion back and a subtraction, which would each
// hold a scheduler's FP64 unit for 64 cycles.  |x| outside 2^-60 .. 2^110
// (zero, thrown to infinity) takes those.
__device__ __forceinline__ void split2(double x, float &hi, float &lo) {
    const uint64_t bits = (uint64_t)__double_as_longlong(x), a = bits & 0x7FFFFFFFFFFFFFFFull;
    const uint32_t e = (uint32_t)(a >> 52);
    if (e - 963u >= 170u) {
        hi = __double2float_rn(x);
        lo = __double2float_rn(__dsub_rn(x, (double)hi));
        return;
    }
    const uint32_t sign = (uint32_t)(bits >> 32) & 0x80000000u;
    // to nearest, ties to even, at bit 29
    const uint64_t b = (a + 0x0FFFFFFFull + ((a >> 29) & 1ull)) >> 29;
    const int r = (int)((uint32_t)a - ((uint32_t)b << 29));  // the remainder, in units of 2^(e - 1075)
    hi = __uint_as_float(((uint32_t)b - 0x1C0000000ull) | sign);
    lo = __int2float_rn(r) * __uint_as_float(((e - 948u) << 23) | sign);
}

// rc2 rounded up to FP32 (host).
inline float round_up_f32(double v) {
    const float f = (float)v;
    return ((double)f < v) ? std::nextafterf(f, INFINITY) : f;
}

// Bound of the FP32 pair filter for particle i at hi position (xh, yh):
// the filter passes pair (i, j) iff |p_j|^2 - 2 p_i.p_j < rc^2 - |p_i|^2 +
// margin, evaluated in FP32 on the hi parts.  The margin 2^-17 (|p_i| + rc)^2
// is ~10x the worst FP32 rounding of that expanded form plus the hi/lo split
// error for any pair within rc of i, so no pair the reference keeps is
// filtered out.  Evaluated in FP32 with every operation rounded in the
// direction that keeps the result an upper bound of the exact value of
// rc^2 - |p_i|^2 + 2^-17 (|p_i| + rc)^2 (|p_i|^2 rounded down where it is
// subtracted, up where it feeds the margin), so the bound can only be
// looser, by a few FP32 ulps of |p_i|^2 -- ~1% of the margin.
__device__ __forceinline__ float filter_threshold(float xh, float yh, float rcf) {  // rcf >= rc^2
    const float a2_dn = __fmaf_rd(xh, xh, __fmul_rd(yh, yh));  // <= |p_i|^2
    const float a2_up = __fmaf_ru(xh, xh, __fmul_ru(yh, yh));  // >= |p_i|^2
    const float pf = __fadd_ru(__fsqrt_ru(a2_up), __fsqrt_ru(rcf));  // >= |p_i| + rc
    const float margin = __fmul_ru(__fmul_ru(pf, pf), 7.62939453125e-6f);
    return __fadd_ru(__fsub_ru(rcf, a2_dn), margin);
}

// Programmatic dependent launch: a kernel launched with the programmatic-
// serialization attribute may be scheduled while its predecessor in the
// stream is still running.  pdl_wait() blocks until the predecessor grid has
// completed and its writes are visible, so every such kernel calls it before
// its first global memory access (a no-op for a kernel launched without the
// attribute).  No kernel here triggers its dependents early
// (griddepcontrol.launch_dependents after the wait): measured on the disk16k
// step sequence it made calm steps 25% slower (0.138 -> 0.172 ms), the next
// kernel's early blocks competing with the running grid's.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Starts bringing a global-memory line into L1 (no data returned, no fault on
// the address being read later by this thread).
__device__ __forceinline__ void prefetch_l1(const void *p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }

__device__ __forceinline__ void write_stage_position(const CloudDev &c, int b, int i, double xs, double ys,
                                                     float rc2_up) {
    c.px[b][i] = xs;
    c.py[b][i] = ys;
    float xh, xl, yh, yl;
    split2(xs, xh, xl);
    split2(ys, yh, yl);
    const double q = c.q[i];
    c.pa[b][i] = make_float4(xh, yh, fmaf(yh, yh, xh * xh), __double2float_rn(q));
    c.pb[b][i] = make_float4(xl, yl, -filter_threshold(xh, yh, rc2_up), 0.0f);
}
__device__ __forceinline__ void write_stage_position(const CloudDev &c, int b, int i, double xs, double ys) {
    write_stage_position(c, b, i, xs, ys, c.rc2_up);
}

// Neither infinite nor NaN, by the exponent bits (a comparison holds the FP64 unit).
__device__ __forceinline__ bool finite64(double v) { return ((uint32_t)__double2hiint(v) & 0x7FF00000u) != 0x7FF00000u; }

// base + inc/2: the product is exact, so one fma is the reference's two operations.
__device__ __forceinline__ double half_step(double base, double inc) { return fma(0.5, inc, base); }

// Position set 1 (x2, y2) of particle i: the step's midpoint for time step dt.
__device__ __forceinline__ void write_midpoint(const CloudDev &c, int i, double x, double y, double vx, double vy,
                                               double dt) {
    write_stage_position(c, 1, i, half_step(x, __dmul_rn(dt, vx)), half_step(y, __dmul_rn(dt, vy)));
}

// The box of a 32-particle group from its lanes' FP32 positions; lane 0
// stores it, every lane returns it.
__device__ __forceinline__ float4 store_group_box(float4 *gbox, bool live, float xh, float yh, bool store) {
    float x0 = live ? xh : INFINITY, y0 = live ? yh : INFINITY;
    float x1 = live ? xh : -INFINITY, y1 = live ? yh : -INFINITY;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        x0 = fminf(x0, __shfl_xor_sync(0xffffffffu, x0, o));
        y0 = fminf(y0, __shfl_xor_sync(0xffffffffu, y0, o));
        x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, o));
        y1 = fmaxf(y1, __shfl_xor_sync(0xffffffffu, y1, o));
    }
    if ((threadIdx.x & 31) == 0 && store) *gbox = make_float4(x0, y0, x1, y1);
    return make_float4(x0, y0, x1, y1);
}

// A padding particle in every position set.
__device__ __forceinline__ void write_padding(const CloudDev &c, int i) {
    for (int b = 0; b < 4; b++) {
        c.px[b][i] = (double)kPadPosition;
        c.py[b][i] = (double)kPadPosition;
        c.pa[b][i] = make_float4(kPadPosition, kPadPosition, kPadPosition * kPadPosition, 0.0f);
        c.pb[b][i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
}

// Reference cutoff decision for one pair, bit for bit:
// r = sqrt(dx*dx + dy*dy) (no fused multiply-add, SSE4.2 has none),
// kappa*r < 10 (ShieldedCoulombForce.cpp:144-147, 175-178).
__host__ __device__ __forceinline__ bool ref_in_cutoff(double dx, double dy, double kappa, double &r,
                                                       double &a) {
#ifdef __CUDA_ARCH__
    r = __dsqrt_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)));
    a = __dmul_rn(r, kappa);
#else
    r = std::sqrt(dx * dx + dy * dy);
    a = r * kappa;
#endif
    return a < 10.0;
}

// Thermal kick of particle i at set e of the running pass (zero when the
// thermal force is off).
__device__ __forceinline__ double2 stage_thermal(const StageParams &P, const ForceParams &f, int i, int e) {
    double tx = 0.0, ty = 0.0;
    if (f.flags & kThermal) {
        thermal_kick(f, (uint32_t)P.c.orig[i], pass_step_index(P), thermal_stage(P, e), tx, ty);
    }
    return make_double2(tx, ty);
}

// DrivingForce::waveNum, angFreq (DrivingForce.cpp:14-15)
constexpr double kWaveNum = 2.0 * 3.14159265358979323846 / 0.002;
constexpr double kAngFreq = 2.0 * 3.14159265358979323846 * 10.0;

// One particle's per-particle forces, each added as the reference's force()
// adds into forceX/forceY (plusEqual_pd / minusEqual_pd); every FP64
// operation is an explicit round-to-nearest intrinsic so nothing is fused.
struct ParticleAt {
    double x, y, vx, vy, q, m;
};

// ConfinementForce::force (ConfinementForce.cpp:48-54), one axis
__device__ __forceinline__ double add_confinement(const ForceParams &f, double q, double p, double F) {
    return __dadd_rn(F, __dmul_rn(__dmul_rn(q, f.confine), p));
}

// DragForce::force (DragForce.cpp:49-55) with dragConst, one axis
__device__ __forceinline__ double add_drag(double dragConst, double m, double v, double F) {
    return __dadd_rn(F, __dmul_rn(__dmul_rn(m, dragConst), v));
}

// sqrt(x*x + y*y) without contraction (length_pd, VectorCompatibility.h:290-292)
__device__ __forceinline__ double radius_of(const ParticleAt &s) {
    return __dsqrt_rn(__dadd_rn(__dmul_rn(s.x, s.x), __dmul_rn(s.y, s.y)));
}

// The terms of the per-particle forces that depend on the position (and the
// force time) alone, each to be added to (or, Rotational, x: subtracted from)
// the force where the reference adds it: ConfinementVoid's second term
// (ConfinementForceVoid.cpp:13-17, 48-55), Driving (DrivingForce.cpp:52-61),
// Rotational (RotationalForce.cpp:50-66), Electric (ElectricForce.cpp:48-62),
// VertElectric (VertElectricForce.cpp:47-53).  They are the expensive ones (FP64
// exp, sin, sqrt, divisions), so a warp per position set computes them while
// the pair sums are under way.
struct PositionTerms {
    double voidx, voidy, drive, rotx, roty, elecx, elecy, vert;
};
// Part `part` of kTermParts of them (fields of T); the parts are about equally
// long chains of FP64 operations, for as many warps.
constexpr int kTermParts = 4;
__device__ __forceinline__ void position_terms(PositionTerms &T, int part, const ForceParams &f, double x, double y,
                                               double q, double t) {
    const long long fl = f.flags;
    auto radius = [&] { return __dsqrt_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y))); };  // length_pd (VectorCompatibility.h:290-292)
    if (part == 0 && (fl & kConfinementVoid)) {
        const double r = radius();
        const double decayV = __dmul_rn(q, -f.void_decay);
        const double expR = __ddiv_rn(exp(__dmul_rn(r, -f.void_decay)), r);
        T.voidx = __dmul_rn(__dmul_rn(decayV, expR), x);
        T.voidy = __dmul_rn(__dmul_rn(decayV, expR), y);
    }
    if (part == 1 && (fl & kDriving)) {
        // the stored driveConst is -drive_const (DrivingForce.h:17-18)
        const double distV = __dsub_rn(x, f.drive_shift);
        const double sinArg = __dsub_rn(__dmul_rn(x, kWaveNum), __dmul_rn(t, kAngFreq));
        const double expArg = __ddiv_rn(__dsub_rn(distV, distV), f.drive_const);
        T.drive = __dmul_rn(__dmul_rn(sin(sinArg), exp(expArg)), f.drive_amplitude);
    }
    if (part == 2) {
        if (fl & kRotational) {
            const double r = radius();
            const bool in = r > f.rot_rmin && r < f.rot_rmax;
            T.rotx = in ? __ddiv_rn(__dmul_rn(f.rot_const, y), r) : 0.0;
            T.roty = in ? __ddiv_rn(__dmul_rn(f.rot_const, x), r) : 0.0;
        }
        if (fl & kVertElectric) T.vert = __dmul_rn(__dmul_rn(q, f.vert_electric), exp(__ddiv_rn(y, f.vert_decay)));
    }
    if (part == 3 && (fl & kElectric)) {
        const double eV = __dmul_rn(__dmul_rn(q, f.electric), exp(__ddiv_rn(radius(), -f.electric_radius)));
        T.elecx = __dmul_rn(eV, x);
        T.elecy = __dmul_rn(eV, y);
    }
}

// Axis ax of the total force on a particle at set e of the running pass, every enabled
// force added in the reference driver's order (driver.cpp:372-402):
// Confinement, ConfinementVoid, Drag, Driving, Magnetic (MagneticForce.cpp:
// 48-54), RectConfinement (RectConfinementForce.cpp:50-59), Rotational,
// ShieldedCoulomb (the pair sum fp), Thermal, ThermalLocalized
// (ThermalForceLocalized.cpp:124-133), TimeVaryingDrag
// (TimeVaryingDragForce.cpp:11-40), TimeVaryingThermal
// (TimeVaryingThermalForce.cpp:14-42), Electric, Gravitational
// (GravitationalForce.cpp:46-50), VertElectric.  T: position_terms at (s.x, s.y).
__device__ __forceinline__ double total_force(const StageParams &P, const ForceParams &f, int i, int e, int ax,
                                              const ParticleAt &s, const PositionTerms &T, double fp) {
    const long long fl = f.flags;
    const double p = ax ? s.y : s.x, v = ax ? s.vy : s.vx;
    double F = 0.0;
    if (fl & kConfinement) F = add_confinement(f, s.q, p, F);
    if (fl & kConfinementVoid) F = __dadd_rn(add_confinement(f, s.q, p, F), ax ? T.voidy : T.voidx);
    if (fl & kDrag) F = add_drag(-f.gamma, s.m, v, F);  // dragConst = -gamma (DragForce.h:16-17)
    if ((fl & kDriving) && ax == 0) F = __dadd_rn(F, T.drive);
    if (fl & kMagnetic) {
        const double qB = __dmul_rn(s.q, f.magnetic);
        F = ax ? __dsub_rn(F, __dmul_rn(qB, s.vx)) : __dadd_rn(F, __dmul_rn(qB, s.vy));
    }
    if (fl & kRectConfinement) F = __dadd_rn(F, __dmul_rn(__dmul_rn(s.q, ax ? f.confine_y : f.confine_x), p));
    if (fl & kRotational) F = ax ? __dadd_rn(F, T.roty) : __dsub_rn(F, T.rotx);
    if (fl & kShieldedCoulomb) F = __dadd_rn(F, fp);
    if (fl & kThermal) {
        const double2 k = stage_thermal(P, f, i, e);
        F = __dadd_rn(F, ax ? k.y : k.x);
    }
    if (fl & kThermalLocalized) {
        const double heat = (radius_of(s) < f.heat_radius) ? f.heat_in : f.heat_out;
        double tx, ty;
        thermal_draw(f, (uint32_t)P.c.orig[i], pass_step_index(P), thermal_stage(P, e) + 16, heat, tx, ty);
        F = __dadd_rn(F, ax ? ty : tx);
    }
    if (fl & (kTimeVaryingDrag | kTimeVaryingThermal)) {
        const double t = stage_time(P, e);
        if (fl & kTimeVaryingDrag) F = add_drag(-__dadd_rn(__dmul_rn(f.drag_scale, t), f.drag_offset), s.m, v, F);
        if (fl & kTimeVaryingThermal) {
            double tx, ty;
            thermal_draw(f, (uint32_t)P.c.orig[i], pass_step_index(P), thermal_stage(P, e) + 32,
                         __dadd_rn(__dmul_rn(f.heat_scale, t), f.heat_offset), tx, ty);
            F = __dadd_rn(F, ax ? ty : tx);
        }
    }
    if (fl & kElectric) F = __dadd_rn(F, ax ? T.elecy : T.elecx);
    if ((fl & kGravitational) && ax) F = __dadd_rn(F, __dmul_rn(s.m, f.gravity));
    if ((fl & kVertElectric) && ax) F = __dadd_rn(F, T.vert);
    return F;
}

// The same for one axis of the forces in kBasicForces (their axes are
// independent), the same operations in the same order.
__device__ __forceinline__ double axis_force(const ForceParams &f, int ax, double x, double v, double q, double m,
                                             double fp, double therm) {
    const long long fl = f.flags;
    double F = (fl & kConfinement) ? __dmul_rn(__dmul_rn(q, f.confine), x) : 0.0;
    if (fl & kDrag) F = __dadd_rn(F, __dmul_rn(__dmul_rn(m, -f.gamma), v));
    if (fl & kRectConfinement) F = __dadd_rn(F, __dmul_rn(__dmul_rn(q, ax ? f.confine_y : f.confine_x), x));
    if (fl & kShieldedCoulomb) F = __dadd_rn(F, fp);
    if (fl & kThermal) F = __dadd_rn(F, therm);
    return F;
}

// a / b given rb = 1/b correctly rounded: one residual correction of a rb, 3 FP64
// instructions instead of the ~9 of a division.  Correctly rounded wherever a rb
// is within one ulp of a/b (Markstein's theorem); the product alone only bounds
// that by 1.5, but of 1.6e9 quotients tried, the corners next to powers of two
// among them, every product was within one ulp and every result that of the
// division (3 and 6 as divisors too).  Zero, tiny, huge and non-finite values
// take the division itself.
__device__ __forceinline__ double div_by(double a, double b, double rb) {
    const double q = __dmul_rn(a, rb);
    const uint32_t ea = ((uint32_t)__double2hiint(a) >> 20) & 0x7FFu, eq = ((uint32_t)__double2hiint(q) >> 20) & 0x7FFu;
    if (ea - 256u >= 1536u || eq - 256u >= 1536u) return __ddiv_rn(a, b);
    return fma(fma(-b, q, a), rb, q);
}
constexpr double kThird = 1.0 / 3.0, kSixth = 1.0 / 6.0;

// One component of a particle's step, in the reference's operations (products
// with 0.5 and 2 are exact, so their sums are one fma each): stage increments
// k = (dt*F)/m, l = dt*V_stage (Runge_Kutta4.cpp:32-104), the CacheOperator
// values (CacheOperator.cpp:28-73), after stage 4 the combine v += (k1 +
// (2*(k2+k3) + k4))/6 (Runge_Kutta4.cpp:107-133, 147-151); RK2's second stage
// ends the step with v += k2, x += l2 (Runge_Kutta2.cpp:68-75).
__device__ __forceinline__ double rk4_sum(double base, double a1, double a2, double a3, double a4) {
    const double s = __dadd_rn(a1, fma(__dadd_rn(a2, a3), 2.0, a4));
    return __dadd_rn(base, div_by(s, 6.0, kSixth));
}

}  // namespace dm
