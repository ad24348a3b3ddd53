// dm_adjoint.cuh -- forces and their vector-Jacobian product for the
// differentiable rollout, in FP64 or FP32-compensated pair arithmetic.
//
// Clouds are concatenated; cloud c owns particles [off_c, off_c + n_c) and
// its own kappa, confinement and drag.  For particle k with force adjoint
// a_k = dL/dF_k (a 2-vector) the VJP kernel produces
//   g_pos[k] = sum_j [ g (a_k - a_j) + h d (d . (a_k - a_j)) ] + q_k k_c a_k
//              (+ rect confinement (q c_x a_x, q c_y a_y))
//   g_vel[k] = -gamma m_k a_k                                    (drag)
//   g_q[k]   = (1/q_k) sum_j F_kj . (a_k - a_j) + k_c p_k . a_k  (dL/dq_k)
//   g_kap[k] = a_k . sum_j (dg/dkappa) d                          (per particle)
//   g_kc[k]  = q_k p_k . a_k                                       (per particle)
// with d = p_k - p_j, F_kj = g(r) d the pair force and, for kappa*r < 10,
//   g(r) = C q_k q_j (1 + kappa r) e^{-kappa r} / r^3,
//   h(r) = g'(r)/r = -g(r) (kappa^2/(1 + kappa r) + 3/r^2),   [since
//          d ln g/dr = -kappa^2 r/(1 + kappa r) - 3/r]
//   dg/dkappa = -C q_k q_j kappa e^{-kappa r} / r.
// This uses that dF_i/dp_i = sum_j G_ij, dF_i/dp_j = -G_ij with the symmetric
// G_ij = g I + h d d^T, so sum_i (dF_i/dp_k)^T a_i = sum_j G_kj (a_k - a_j).
// The cutoff is the reference's (ShieldedCoulombForce.cpp:147); the force is
// discontinuous there and its jump is not differentiated (measure zero).
#pragma once

#include "dm_pair.cuh"

namespace dm {

struct AdjCloud {
    int off, n;
    long long flags;
    double kappa, confine, confine_x, confine_y, gamma;
    double rc2;
    float rc2_lo, rc2_hi;  // FP32 certain-in / certain-out bounds on r^2
    float rc2_up;          // rc2 rounded up
    float kappa_f, kappa2_f;
    float kl2e_hi, kl2e_lo;  // kappa*log2(e) as a float pair (SFU exponential)
    float nkl2e;             // -kappa*log2(e): e^{-kappa r} = 2^{nkl2e r} (packed pair terms)
    Yukawa64 y64;
};

constexpr int kAdjThreads = 128;
constexpr int kAdjTile = 256;

// FP32-compensated pair loop over one shared-memory j tile: positions as
// float pairs (hi, lo) so the differences keep ~2^-24 relative accuracy,
// pair terms in FP32, summed plainly over groups of four j and each group
// added to Kahan sums; pairs within 4e-6 of the cutoff in r^2 are decided by
// the reference's FP64 test on the FP64 positions.  e^{-kappa r} on the SFU
// with the rounding residue of kappa r restored (exp_neg_kr), 1/(1 + kappa r)
// from the fast reciprocal: a few ulp per pair term, far below the rounding
// of the FP32 pair sums themselves.
template <int MODE>
__device__ __forceinline__ void adj_tile_fp32c(const AdjCloud &d, const float4 *sp,
                                               const float4 *sa, int cnt, int jbase, int li, float xh, float yh,
                                               float xl, float yl, float qci, float axi, float ayi,
                                               const double *__restrict__ x, const double *__restrict__ y,
                                               double xi, double yi, float (&s)[4], float (&c)[4]) {
    constexpr int NS = MODE == 0 ? 2 : 4;
    for (int e0 = 0; e0 < cnt; e0 += 4) {
        float t[NS];
#pragma unroll
        for (int k = 0; k < NS; k++) t[k] = 0.0f;
        const int e1 = min(cnt, e0 + 4);
        for (int e = e0; e < e1; e++) {
            const float4 P = sp[e];
            const float dx = (xh - P.x) + (xl - P.z);
            const float dy = (yh - P.y) + (yl - P.w);
            const float r2 = fmaf(dx, dx, dy * dy);
            if (!(r2 < d.rc2_hi)) continue;
            if (jbase + e == li) continue;
            if (!(r2 < d.rc2_lo)) {
                const int j = d.off + jbase + e;
                double r, a;
                if (!ref_in_cutoff(__dsub_rn(xi, x[j]), __dsub_rn(yi, y[j]), d.kappa, r, a)) continue;
            }
            float w = rsqrtf(r2);  // 1/r, one Newton step
            w = fmaf(0.5f * fmaf(-(r2 * w), w, 1.0f), w, w);
            const float r = r2 * w;
            const float kr = d.kappa_f * r;
            const float ex = exp_neg_kr(r, d.kl2e_hi, d.kl2e_lo);
            const float4 A = sa[e];  // (q_j, a_j.x, a_j.y, -)
            const float qq = qci * A.x;
            const float g = (qq * (1.0f + kr)) * ex * ((w * w) * w);
            if constexpr (MODE == 0) {
                t[0] = fmaf(g, dx, t[0]);
                t[1] = fmaf(g, dy, t[1]);
            } else {
                const float h = -g * fmaf(d.kappa2_f, __fdividef(1.0f, 1.0f + kr), 3.0f * (w * w));
                const float bx = axi - A.y, by = ayi - A.z;
                const float dd = fmaf(dx, bx, dy * by);
                const float hd = h * dd;
                t[0] += fmaf(hd, dx, g * bx);
                t[1] += fmaf(hd, dy, g * by);
                t[2] = fmaf(g, dd, t[2]);
                t[NS - 1] = fmaf(-(qq * d.kappa_f) * ex * w, fmaf(axi, dx, ayi * dy), t[NS - 1]);
            }
        }
#pragma unroll
        for (int k = 0; k < NS; k++) kahan_add(s[k], c[k], t[k]);
    }
}

// One thread per particle i, j of the same cloud staged through shared
// memory.  MODE 0: forces (total F and pair-only Fp).  MODE 1: VJP.
// FP32-compensated pair arithmetic (FP64: adj_group_fp64).
struct AdjOnce {
    const double *x, *y, *vx, *vy, *q, *m;
    const double *ax, *ay;  // MODE 1: force adjoint
    double *o[7];
};

// The outputs of particle i from its pair sums S (C q_i included; S[2] is
// sum_j F_ij . (a_i - a_j), S[3] the kappa sum).
template <int MODE>
__device__ __forceinline__ void adj_once_outputs(const AdjCloud &d, const AdjOnce &A, int i, const double (&S)[4]) {
    const double xi = A.x[i], yi = A.y[i], qi = A.q[i], xv = A.vx[i], yv = A.vy[i], mi = A.m[i];
    if (MODE == 0) {
        double fx = 0.0, fy = 0.0;
        if (d.flags & kConfinement) { fx += qi * d.confine * xi; fy += qi * d.confine * yi; }
        if (d.flags & kDrag) { fx += -d.gamma * mi * xv; fy += -d.gamma * mi * yv; }
        if (d.flags & kRectConfinement) { fx += qi * d.confine_x * xi; fy += qi * d.confine_y * yi; }
        A.o[0][i] = fx + S[0];   // total force
        A.o[1][i] = fy + S[1];
        if (A.o[2]) A.o[2][i] = S[0];  // pair force only
        if (A.o[3]) A.o[3][i] = S[1];
    } else {
        const double axi = A.ax[i], ayi = A.ay[i];
        double gx = S[0], gy = S[1], gq = (qi != 0.0) ? S[2] / qi : 0.0, gkc = 0.0;
        if (d.flags & kConfinement) {
            gx += qi * d.confine * axi;
            gy += qi * d.confine * ayi;
            gq += d.confine * (xi * axi + yi * ayi);
            gkc = qi * (xi * axi + yi * ayi);
        }
        if (d.flags & kRectConfinement) {
            gx += qi * d.confine_x * axi;
            gy += qi * d.confine_y * ayi;
            gq += d.confine_x * xi * axi + d.confine_y * yi * ayi;
        }
        const double gv = (d.flags & kDrag) ? -d.gamma * mi : 0.0;
        A.o[0][i] = gx;          // dL/dp (through the forces)
        A.o[1][i] = gy;
        A.o[2][i] = gv * axi;    // dL/dv (through drag)
        A.o[3][i] = gv * ayi;
        A.o[4][i] = gq;          // dL/dq_i
        A.o[5][i] = S[3];        // dL/dkappa contribution of particle i
        A.o[6][i] = gkc;         // dL/dk_c contribution of particle i
    }
}

template <int MODE>
__global__ void __launch_bounds__(kAdjThreads) adjoint_kernel(const AdjCloud *__restrict__ desc,
                                                              const int *__restrict__ cloud_of_block,
                                                              const int *__restrict__ tile_of_block, const AdjOnce A,
                                                              double coulomb) {
    __shared__ float4 sp[kAdjTile], sa[kAdjTile];
    const AdjCloud d = desc[cloud_of_block[blockIdx.x]];
    const int li = tile_of_block[blockIdx.x] * kAdjThreads + threadIdx.x;  // index within the cloud
    const bool valid = li < d.n;
    const int i = d.off + (valid ? li : 0);
    const double xi = A.x[i], yi = A.y[i];
    const float axf = (MODE == 1 && valid) ? (float)A.ax[i] : 0.0f, ayf = (MODE == 1 && valid) ? (float)A.ay[i] : 0.0f;
    const float xh = (float)xi, yh = (float)yi;
    const float xl = (float)(xi - (double)xh), yl = (float)(yi - (double)yh);
    const float qci = (float)(coulomb * A.q[i]);
    float fs[4] = {0.0f, 0.0f, 0.0f, 0.0f}, fc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    for (int j0 = 0; j0 < d.n && (d.flags & kShieldedCoulomb); j0 += kAdjTile) {
        const int cnt = min(kAdjTile, d.n - j0);
        __syncthreads();
        for (int e = threadIdx.x; e < cnt; e += kAdjThreads) {
            const int j = d.off + j0 + e;
            const double xj = A.x[j], yj = A.y[j];
            const float hx = (float)xj, hy = (float)yj;
            sp[e] = make_float4(hx, hy, (float)(xj - (double)hx), (float)(yj - (double)hy));
            sa[e] = make_float4((float)A.q[j], MODE == 1 ? (float)A.ax[j] : 0.0f, MODE == 1 ? (float)A.ay[j] : 0.0f,
                                0.0f);
        }
        __syncthreads();
        if (valid)
            adj_tile_fp32c<MODE>(d, sp, sa, cnt, j0, li, xh, yh, xl, yl, qci, axf, ayf, A.x, A.y, xi, yi, fs, fc);
    }
    if (!valid) return;
    double S[4];
#pragma unroll
    for (int k = 0; k < 4; k++) S[k] = (double)fs[k] - (double)fc[k];
    adj_once_outputs<MODE>(d, A, i, S);
}

// ===========================================================================
// Fused RK4 step and its adjoint for the differentiable rollout.
//
// One launch per RK4 stage.  Forward (adj_step_fp64, adj_step_fp32c): the pair force at
// the stage's input state, the per-particle forces, and the stage algebra
// of the rollout's RK4 step in FP64 (for s = (x, y, vx, vy) and f(s) =
// (vx, vy, Fx/m, Fy/m)):
//     k_s = dt f(s_s),  s_2 = S + k_1/2, s_3 = S + k_2/2, s_4 = S + k_3,
//     S' = S + (k_1 + ((k_2 + k_3) 2 + k_4)) / 6,
// with the operations in that order (each rounded, nothing contracted).
// Backward (adj_vjp_fp64, adj_vjp_fp32c, stages 4, 3, 2, 1): given lam = dL/dS', the stage
// weights dk_4 = lam/6, dk_3 = lam/3 + mu_4, dk_2 = lam/3 + mu_3/2,
// dk_1 = lam/6 + mu_2/2 with mu_s = J(s_s)^T (dt dk_s), and finally
// dL/dS = lam + mu_1 + mu_2 + mu_3 + mu_4; the parameter gradients
// (dt dk_s)^T df/dtheta are added into per-particle accumulators.  J^T w
// for f is (the force VJP of a = w_v / m) for positions, w_p - gamma w_v
// for velocities.
//
// The kernels read positions split once per particle and stage (AdjSplit: by
// adj_prepare for the first stage of a call, by the epilogue of the stage
// before for the others): FP32 hi and lo parts, |p|^2, the conservative filter
// bound (filter_threshold) and, backward, the FP32 force adjoint.  Splitting in
// every block that reads a particle cost four FP64-pipe conversions each time.
//
// FP32C pair terms: one i per thread, j staged in shared memory as negated
// two-float positions (plus charge and, backward, the j's force adjoint).
// Chunks of 4 j are filtered first (two j per packed FMA); a lane evaluates
// its own hit chunks, two j per packed f32x2 evaluation, the cutoff by a
// select (pairs within 4e-6 of it in r^2 decided by the reference's FP64 test
// on the FP64 positions), plain sums over four j, then Kahan; C q_i applied in
// FP64 per particle.  A chunk that is skipped would have added zeros: the
// first zero after a term may still move a bit between Kahan's sum and its
// correction, later ones change nothing, so a run of skipped chunks is one
// added zero and the filter leaves every bit of the result as it was.
// Where most lanes of a warp hit most chunks the warp takes the chunks one by
// one, all lanes on the same 4 j.
//
// FP64: adj_group_fp64.
// ===========================================================================

constexpr int kAsJ = 512;  // j staged per tile (a multiple of 128)

struct AdjSplit {
    float4 *p;  // xh, yh, |p|^2, -(filter bound)
    float2 *l;  // xl, yl
    float2 *a;  // FP32 force adjoint (backward)
};

struct AdjStepIO {
    const double *x, *y, *vx, *vy;  // the stage's input state s_s
    double *s[4];                   // the step's base state S (stage 4 writes S' over it)
    double *k1[4], *k23[4];         // k_1 and k_2 + k_3
    double *next[4];                // the next stage's input (stages 1-3)
    AdjSplit in, out;               // split positions of this stage's input; of the next's
    const double *q, *m, *invm;     // invm = 1/m
    double dt;
    int stage;
};

struct AdjVjpIO {
    const double *x, *y;            // the stage's input positions
    const double *xn, *yn;          // those of stage s-1 (stages 4-2)
    const double *dk[4];            // dk_s
    double *dkn[4];                 // dk_{s-1} (stages 4-2)
    double *lam[4];                 // dL/dS' in, dL/dS out (stage 1)
    double *mu[3][4];               // mu_4, mu_3, mu_2
    double *gq, *gkappa, *gkc;      // per-particle parameter gradients (added to)
    const double *ax, *ay;          // force adjoint a = dt dk_v / m of stage s
    double *axn, *ayn;              // of stage s-1
    AdjSplit in, out;
    const double *q, *m, *invm;
    double dt;
    int stage;
};

__device__ __forceinline__ float4 adj_split_hi(float xh, float yh, float rc2_up) {
    return make_float4(xh, yh, fmaf(yh, yh, xh * xh), -filter_threshold(xh, yh, rc2_up));
}
__device__ __forceinline__ void adj_store_split(const AdjSplit &o, int i, double x, double y, float rc2_up) {
    float xh, xl, yh, yl;
    split2(x, xh, xl);
    split2(y, yh, yl);
    o.p[i] = adj_split_hi(xh, yh, rc2_up);
    o.l[i] = make_float2(xl, yl);
}

// AdjSplit::p of particle i: as stored, or formed where it is read (calls of
// their own, which keep no scratch; the same values; for a j the bound's
// arithmetic falls away).
struct AdjStoredSplit {
    const float4 *p;
    __device__ __forceinline__ float4 operator()(int i) const { return p[i]; }
};
struct AdjFormedSplit {
    const double *x, *y;
    float rc2_up;
    __device__ __forceinline__ float4 operator()(int i) const {
        return adj_split_hi(__double2float_rn(x[i]), __double2float_rn(y[i]), rc2_up);
    }
};

// Splits positions (x, y); invm (if given) = 1/m; backward (lam given): dk_4 =
// lam/6 and the force adjoint a = dt dk_v / m of stage 4.
struct AdjPrepareIO {
    const double *x, *y, *m;
    AdjSplit out;
    double *invm;
    const double *lam[4];
    double *dk[4];
    double *ax, *ay;
    double dt;
};
static __global__ void __launch_bounds__(kAdjThreads) adj_prepare(const AdjCloud *__restrict__ desc,
                                                                  const int *__restrict__ cloud_of_block,
                                                                  const int *__restrict__ tile_of_block,
                                                                  const AdjPrepareIO R) {
    const AdjCloud &d = desc[cloud_of_block[blockIdx.x]];
    const int li = tile_of_block[blockIdx.x] * kAdjThreads + threadIdx.x;
    if (li >= d.n) return;
    const int i = d.off + li;
    adj_store_split(R.out, i, R.x[i], R.y[i], d.rc2_up);
    if (!R.invm) return;
    const double m = R.m[i], inv = __drcp_rn(m);
    R.invm[i] = inv;
    if (!R.lam[0]) return;
    double a[4];
#pragma unroll
    for (int c = 0; c < 4; c++) {
        a[c] = div_by(R.lam[c][i], 6.0, kSixth);
        R.dk[c][i] = a[c];
    }
    const double ax = div_by(__dmul_rn(R.dt, a[2]), m, inv), ay = div_by(__dmul_rn(R.dt, a[3]), m, inv);
    R.ax[i] = ax;
    R.ay[i] = ay;
    R.out.a[i] = make_float2((float)ax, (float)ay);
}

// Component c (x, y, vx, vy) of particle i's forward stage, pair the pair
// force along the component's axis.  Returns the next stage's value.
__device__ __forceinline__ double adj_step_component(const AdjCloud &d, const AdjStepIO &io, int i, int c,
                                                     double pair) {
    const bool ya = (c & 1) != 0;
    const double v = (ya ? io.vy : io.vx)[i];
    double k;
    if (c < 2) {
        k = __dmul_rn(io.dt, v);
    } else {
        const double xi = (ya ? io.y : io.x)[i], qi = io.q[i], mi = io.m[i];
        double f = 0.0;
        if (d.flags & kConfinement) f += qi * d.confine * xi;
        if (d.flags & kDrag) f += -d.gamma * mi * v;
        if (d.flags & kRectConfinement) f += qi * (ya ? d.confine_y : d.confine_x) * xi;
        f += pair;
        k = __dmul_rn(io.dt, div_by(f, mi, io.invm[i]));
    }
    // halves and doubles are exact: one rounding per operation as written above
    const double base = io.s[c][i];
    double next;
    if (io.stage == 1) {
        io.k1[c][i] = k;
        next = fma(0.5, k, base);
    } else if (io.stage == 2) {
        io.k23[c][i] = k;
        next = fma(0.5, k, base);
    } else if (io.stage == 3) {
        io.k23[c][i] = __dadd_rn(io.k23[c][i], k);
        next = __dadd_rn(base, k);
    } else {
        const double inc = div_by(__dadd_rn(io.k1[c][i], fma(io.k23[c][i], 2.0, k)), 6.0, kSixth);
        next = __dadd_rn(base, inc);
    }
    (io.stage == 4 ? io.s[c] : io.next[c])[i] = next;
    return next;
}

// Component c of particle i's backward stage from its pair sums S (C q_i
// included), and the parameter gradients (c = 2: dq; c = 3: dkappa, dk_c).
// Returns dk_{s-1} of the component (stages 4-2).
__device__ __forceinline__ double adj_vjp_component(const AdjCloud &d, const AdjVjpIO &V, int i, int c,
                                                    const double (&S)[4]) {
    const bool ya = (c & 1) != 0;
    const double xi = V.x[i], yi = V.y[i], qi = V.q[i];
    const double axi = V.ax[i], ayi = V.ay[i], a = ya ? ayi : axi;
    // mu = J^T (dt dk): positions through the forces, velocities through
    // f_pos = v and the drag
    double mu;
    if (c < 2) {
        mu = S[c];
        if (d.flags & kConfinement) mu += qi * d.confine * a;
        if (d.flags & kRectConfinement) mu += qi * (ya ? d.confine_y : d.confine_x) * a;
    } else {
        const double gv = (d.flags & kDrag) ? -d.gamma * V.m[i] : 0.0;
        mu = __dadd_rn(__dmul_rn(V.dt, V.dk[c - 2][i]), gv * a);
    }
    if (c == 2) {
        double gq = (qi != 0.0) ? S[2] / qi : 0.0;
        if (d.flags & kConfinement) gq += d.confine * (xi * axi + yi * ayi);
        if (d.flags & kRectConfinement) gq += d.confine_x * xi * axi + d.confine_y * yi * ayi;
        V.gq[i] += gq;
    } else if (c == 3) {
        V.gkappa[i] += S[3];
        if (d.flags & kConfinement) V.gkc[i] += qi * (xi * axi + yi * ayi);
    }
    const double l = V.lam[c][i];
    double dkn = 0.0;
    if (V.stage == 4) {
        V.mu[0][c][i] = mu;
        dkn = __dadd_rn(div_by(l, 3.0, kThird), mu);
    } else if (V.stage == 3) {
        V.mu[1][c][i] = mu;
        dkn = fma(0.5, mu, div_by(l, 3.0, kThird));
    } else if (V.stage == 2) {
        V.mu[2][c][i] = mu;
        dkn = fma(0.5, mu, div_by(l, 6.0, kSixth));
    } else {
        V.lam[c][i] = __dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(l, mu), V.mu[2][c][i]), V.mu[1][c][i]), V.mu[0][c][i]);
        return 0.0;
    }
    V.dkn[c][i] = dkn;
    return dkn;
}

// The force adjoint of stage s-1 along one axis.
__device__ __forceinline__ double adj_next_force_adjoint(const AdjVjpIO &V, int i, double dkn) {
    return div_by(__dmul_rn(V.dt, dkn), V.m[i], V.invm[i]);
}

// One pair term in FP32 for the slow path (pairs within 4e-6 of the cutoff
// in r^2): 0 outside the cutoff (the reference's FP64 test decides).
__device__ __forceinline__ bool adj_border_in(const AdjCloud &d, const double *x, const double *y, int i, int j) {
    double r, a;
    return ref_in_cutoff(__dsub_rn(x[i], x[j]), __dsub_rn(y[i], y[j]), d.kappa, r, a);
}

// FP32C pair sums of particle li of cloud d over the cloud's j, staged kAsJ
// at a time as chunks of 4 j (one float4 per quantity).  MODE 0: out[0..1] =
// sum_j w_ij (dx, dy) (times C q_i: the pair force).  MODE 1 (a_i, a_j the
// force adjoints): out[0..1] = sum w b + h d (d . b), out[2] = sum w (d . b),
// out[3] = sum q_j e y (a_i . d) (times C q_i: the position VJP, F_ij . (a_i -
// a_j) and, times -kappa, dg/dkappa), with b = a_i - a_j.  j == i is the pair
// with r^2 = 0 exactly (dx = dy = 0), left out by the select.  Every thread of
// the block calls it.
template <int MODE>
__device__ __forceinline__ void adj_pair_sums_fp32c(const AdjCloud &d, int li, bool valid, const double *x,
                                                    const double *y, const double *q, const AdjSplit &in,
                                                    float (&out)[4]) {
    constexpr int NQ = MODE == 0 ? 6 : 8;  // -xh, -yh, |p|^2, -xl, -yl, q (, a_x, a_y)
    constexpr int NC = kAsJ / 4, NWORD = NC / 32;
    __shared__ float4 s_c[NQ][NC];
    constexpr int NS = MODE == 0 ? 2 : 4;
    float sum[NS], cmp[NS];
#pragma unroll
    for (int k = 0; k < NS; k++) sum[k] = cmp[k] = 0.0f;
    const int i = d.off + (valid ? li : 0);
    float4 pi = make_float4(0.0f, 0.0f, 0.0f, INFINITY);
    float2 lo2 = make_float2(0.0f, 0.0f), ai = make_float2(0.0f, 0.0f);
    if (valid) {
        pi = in.p[i];
        lo2 = in.l[i];
        if (MODE == 1) ai = in.a[i];
    }
    const PairI I{dup2(pi.x), dup2(pi.y), dup2(lo2.x), dup2(lo2.y)};
    const float2 px2 = dup2(2.0f * pi.x), py2 = dup2(2.0f * pi.y), nu2 = dup2(pi.w);
    const float2 kap = dup2(d.kappa_f), nkl2e = dup2(d.nkl2e);
    const float2 nk2 = dup2(-d.kappa2_f), m3 = dup2(-3.0f);
    const float2 ax2 = dup2(ai.x), ay2 = dup2(ai.y);
    const float lo = d.rc2_lo, hi = d.rc2_hi;
    float *s_f = reinterpret_cast<float *>(s_c);
    int last = -1;  // this lane's last evaluated chunk, over the whole cloud
    auto add_zero = [&] {
#pragma unroll
        for (int k = 0; k < NS; k++) kahan_add(sum[k], cmp[k], 0.0f);
    };
    int dense = 0;  // words of chunks to take without filtering (the last one filtered was mostly hits)
    for (int j0 = 0; j0 < d.n; j0 += kAsJ) {
        const int cnt = min(kAsJ, d.n - j0);
        const int nch = (cnt + 3) >> 2;
        __syncthreads();
        for (int e = threadIdx.x; e < 4 * nch; e += blockDim.x) {
            float v[NQ];
            if (e < cnt) {
                const int j = d.off + j0 + e;
                const float4 A = in.p[j];
                const float2 B = in.l[j];
                v[0] = -A.x;
                v[1] = -A.y;
                v[2] = A.z;
                v[3] = -B.x;
                v[4] = -B.y;
                v[5] = (float)q[j];
                if (MODE == 1) {
                    const float2 aj = in.a[j];
                    v[NQ - 2] = aj.x;
                    v[NQ - 1] = aj.y;
                }
            } else {  // padding: far away, no charge (a finite, zero term)
                v[0] = v[1] = -kPadPosition;
                v[2] = INFINITY;
                v[3] = v[4] = v[5] = 0.0f;
                if (MODE == 1) v[NQ - 2] = v[NQ - 1] = 0.0f;
            }
#pragma unroll
            for (int k = 0; k < NQ; k++) s_f[k * kAsJ + e] = v[k];  // s_c[k][e/4].{x,y,z,w}[e%4]
        }
        __syncthreads();
        if (!__any_sync(0xffffffffu, valid)) continue;
        // the 4 pairs of chunk c (any c per lane)
        auto chunk = [&](int c) {
            if (j0 / 4 + c != last + 1) add_zero();
            last = j0 / 4 + c;
            float4 Q[NQ];
#pragma unroll
            for (int k = 0; k < NQ; k++)
                if (k != 2) Q[k] = s_c[k][c];
            float2 part[NS];
#pragma unroll
            for (int k = 0; k < NS; k++) part[k] = dup2(0.0f);
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const float2 nxh = h ? make_float2(Q[0].z, Q[0].w) : make_float2(Q[0].x, Q[0].y);
                const float2 nyh = h ? make_float2(Q[1].z, Q[1].w) : make_float2(Q[1].x, Q[1].y);
                const float2 nxl = h ? make_float2(Q[3].z, Q[3].w) : make_float2(Q[3].x, Q[3].y);
                const float2 nyl = h ? make_float2(Q[4].z, Q[4].w) : make_float2(Q[4].x, Q[4].y);
                const float2 qj = h ? make_float2(Q[5].z, Q[5].w) : make_float2(Q[5].x, Q[5].y);
                float2 dx, dy, r2, yy, ex;
                pair2_core(I, nxh, nyh, nxl, nyl, nkl2e, dx, dy, r2, yy, ex);
                bool ina = r2.x < lo && r2.x > 0.0f, inb = r2.y < lo && r2.y > 0.0f;
                // pairs within 4e-6 of the cutoff in r^2: the reference's FP64 test
                if ((r2.x >= lo && r2.x < hi) || (r2.y >= lo && r2.y < hi)) {
                    const int ja = j0 + 4 * c + 2 * h;
                    if (r2.x >= lo && r2.x < hi && ja < d.n) ina = adj_border_in(d, x, y, i, d.off + ja);
                    if (r2.y >= lo && r2.y < hi && ja + 1 < d.n) inb = adj_border_in(d, x, y, i, d.off + ja + 1);
                }
                // q_j e^{-kappa r} and 1/r, both 0 outside the cutoff and for j == i
                // (where r = 0 made them non-finite), so every term below is 0 there
                float2 qe = mul2(qj, ex);
                qe.x = ina ? qe.x : 0.0f;
                qe.y = inb ? qe.y : 0.0f;
                yy.x = ina ? yy.x : 0.0f;
                yy.y = inb ? yy.y : 0.0f;
                const float2 y2 = mul2(yy, yy);
                const float2 t = add2(yy, kap);
                const float2 ww = mul2(qe, mul2(y2, t));  // g / (C q_i)
                if (MODE == 0) {
                    part[0] = fma2(ww, dx, part[0]);
                    part[1] = fma2(ww, dy, part[1]);
                } else {
                    const float4 QX = Q[NQ - 2], QY = Q[NQ - 1];
                    const float2 ajx2 = h ? make_float2(QX.z, QX.w) : make_float2(QX.x, QX.y);
                    const float2 ajy2 = h ? make_float2(QY.z, QY.w) : make_float2(QY.x, QY.y);
                    // h / (C q_i) = -q_j e y^3 (kappa^2 + 3 y (y + kappa))
                    const float2 hv = mul2(mul2(qe, mul2(y2, yy)), fma2(mul2(yy, m3), t, nk2));
                    const float2 bx = add2(ax2, make_float2(-ajx2.x, -ajx2.y));
                    const float2 by = add2(ay2, make_float2(-ajy2.x, -ajy2.y));
                    const float2 dd = fma2(dx, bx, mul2(dy, by));
                    const float2 aid = fma2(ax2, dx, mul2(ay2, dy));
                    const float2 hdd = mul2(hv, dd);
                    part[0] = fma2(ww, bx, fma2(hdd, dx, part[0]));
                    part[1] = fma2(ww, by, fma2(hdd, dy, part[1]));
                    part[2] = fma2(ww, dd, part[2]);
                    part[3] = fma2(mul2(qe, yy), aid, part[3]);
                }
            }
#pragma unroll
            for (int k = 0; k < NS; k++) kahan_add(sum[k], cmp[k], part[k].x + part[k].y);
        };
        for (int w = 0; w < NWORD; w++) {
            const int c0 = 32 * w, cn = min(32, nch - c0);
            if (cn <= 0) break;
            uint32_t m = 0u;
            if (dense == 0) {
#pragma unroll 4
                for (int u = 0; u < cn; u++) {
                    const float4 X = s_c[0][c0 + u], Y = s_c[1][c0 + u], B = s_c[2][c0 + u];
                    const float2 d01 = fma2(px2, make_float2(X.x, X.y),
                                            fma2(py2, make_float2(Y.x, Y.y), add2(make_float2(B.x, B.y), nu2)));
                    const float2 d23 = fma2(px2, make_float2(X.z, X.w),
                                            fma2(py2, make_float2(Y.z, Y.w), add2(make_float2(B.z, B.w), nu2)));
                    const uint32_t sg = __float_as_uint(d01.x) | __float_as_uint(d01.y) | __float_as_uint(d23.x) |
                                        __float_as_uint(d23.y);
                    m = __funnelshift_l(sg, m, 1);  // newest chunk in bit 0
                }
                // chunk c0 + u is bit u from here on; a lane without a particle
                // (bound INFINITY) or pairs all NaN may set bits: no matter
                m = __brev(m) >> (32 - cn);
                if (__reduce_add_sync(0xffffffffu, __popc(m)) >= 16 * cn) dense = 4;
            }
            if (dense) {
                dense--;
                for (int u = 0; u < cn; u++) chunk(c0 + u);
            } else {
                while (m) {
                    chunk(c0 + __ffs(m) - 1);
                    m &= m - 1u;
                }
            }
        }
    }
    if (last != ((d.n + 3) >> 2) - 1) add_zero();
#pragma unroll
    for (int k = 0; k < 4; k++) out[k] = (k < NS) ? sum[k] - cmp[k] : 0.0f;
}

// Forward stage of the fused RK4 step, FP32C (one thread per particle).
static __global__ void __launch_bounds__(kAdjThreads) adj_step_fp32c(const AdjCloud *__restrict__ desc,
                                                                     const int *__restrict__ cloud_of_block,
                                                                     const int *__restrict__ tile_of_block,
                                                                     const AdjStepIO io, double coulomb) {
    const AdjCloud d = desc[cloud_of_block[blockIdx.x]];
    const int li = tile_of_block[blockIdx.x] * kAdjThreads + threadIdx.x;
    const bool valid = li < d.n;
    const int i = d.off + (valid ? li : 0);
    double px = 0.0, py = 0.0;
    if (d.flags & kShieldedCoulomb) {
        float o[4];
        adj_pair_sums_fp32c<0>(d, li, valid, io.x, io.y, io.q, io.in, o);
        const double cq = __dmul_rn(coulomb, io.q[i]);
        px = __dmul_rn(cq, (double)o[0]);
        py = __dmul_rn(cq, (double)o[1]);
    }
    if (!valid) return;
    const double nx = adj_step_component(d, io, i, 0, 0.0), ny = adj_step_component(d, io, i, 1, 0.0);
    adj_step_component(d, io, i, 2, px);
    adj_step_component(d, io, i, 3, py);
    if (io.stage < 4) adj_store_split(io.out, i, nx, ny, d.rc2_up);
}

// Backward stage, FP32C (one thread per particle).
static __global__ void __launch_bounds__(kAdjThreads) adj_vjp_fp32c(const AdjCloud *__restrict__ desc,
                                                                    const int *__restrict__ cloud_of_block,
                                                                    const int *__restrict__ tile_of_block,
                                                                    const AdjVjpIO V, double coulomb) {
    const AdjCloud d = desc[cloud_of_block[blockIdx.x]];
    const int li = tile_of_block[blockIdx.x] * kAdjThreads + threadIdx.x;
    const bool valid = li < d.n;
    const int i = d.off + (valid ? li : 0);
    double S[4] = {0.0, 0.0, 0.0, 0.0};
    if (d.flags & kShieldedCoulomb) {
        float o[4];
        adj_pair_sums_fp32c<1>(d, li, valid, V.x, V.y, V.q, V.in, o);
        const double cq = __dmul_rn(coulomb, V.q[i]);
        S[0] = __dmul_rn(cq, (double)o[0]);
        S[1] = __dmul_rn(cq, (double)o[1]);
        S[2] = __dmul_rn(cq, (double)o[2]);
        S[3] = __dmul_rn(__dmul_rn(-d.kappa, cq), (double)o[3]);
    }
    if (!valid) return;
    adj_vjp_component(d, V, i, 0, S);
    adj_vjp_component(d, V, i, 1, S);
    const double kx = adj_vjp_component(d, V, i, 2, S), ky = adj_vjp_component(d, V, i, 3, S);
    if (V.stage > 1) {
        const double ax = adj_next_force_adjoint(V, i, kx), ay = adj_next_force_adjoint(V, i, ky);
        V.axn[i] = ax;
        V.ayn[i] = ay;
        V.out.a[i] = make_float2((float)ax, (float)ay);
        adj_store_split(V.out, i, V.xn[i], V.yn[i], d.rc2_up);
    }
}

// ---------------------------------------------------------------------------
// FP64: one 32-particle group of a cloud per tile, a cluster of S blocks of
// four warps per tile.  The cloud's j groups are dealt to the 4 S warps; each
// is filtered in FP32 and its hits evaluated in FP64 with full warps
// (dm_fp64.cuh), or, where most of the 32 x 32 pairs are hits, lane by lane
// (every lane its own i, all on the same j: no list, the sums by FMA).  The
// four warps of the cluster's first block then take one component each of the
// particles' stage epilogue.  Bound by the FP64 pipe: 20 (forward) and 35
// (backward) FP64 instructions per pair, 2 and 4 more to add up a listed hit.
// ---------------------------------------------------------------------------
constexpr int kAdjWarps = 4;

template <int NS>
struct AdjGroupSmem {
    HitWarp<HitResult<NS>> w[kAdjWarps];
    double tab[kExp2Size];
    double ix[32], iy[32], iax[32], iay[32];
    double acc[kAdjWarps][NS][32];
    double red[NS][32];
    double xch[2][32];
};

// The pair's terms of MODE 0 (2 sums) or MODE 1 (4 sums), as listed at
// adj_pair_sums_fp32c, added to s by FMA; `in`: inside the cutoff and j != i.
template <int MODE>
__device__ __forceinline__ void adj_pair64(const Yukawa64 &K, const double *tab, double dx, double dy, double qj,
                                           double aix, double aiy, double ajx, double ajy, bool use,
                                           double (&s)[MODE == 0 ? 2 : 4]) {
    const double r2 = fma(dx, dx, __dmul_rn(dy, dy));
    use = use && in_cutoff64(dx, dy, r2, K);
    Yukawa64At A;
    if (yukawa64_odd(r2)) A = yukawa64_general(r2, K.kappa);
    else A = yukawa64(r2, K, tab);
    // q_j e^{-kappa r} / r is 0 for a pair that does not count; its 1/r must
    // stay finite (j == i)
    const double y = use ? A.y : 1.0;
    const double qy = use ? __dmul_rn(__dmul_rn(qj, A.ex), A.y) : 0.0;
    const double t = __dmul_rn(y, __dadd_rn(y, K.kappa));
    const double w = __dmul_rn(qy, t);
    if constexpr (MODE == 0) {
        s[0] = fma(w, dx, s[0]);
        s[1] = fma(w, dy, s[1]);
    } else {
        // h / (C q_i) = -q_j e y^3 (kappa^2 + 3 y (y + kappa))
        const double nh = __dmul_rn(__dmul_rn(qy, __dmul_rn(y, y)), fma(3.0, t, __dmul_rn(K.kappa, K.kappa)));
        const double bx = __dsub_rn(aix, ajx), by = __dsub_rn(aiy, ajy);
        const double dd = fma(dx, bx, __dmul_rn(dy, by));
        const double hd = __dmul_rn(nh, dd);
        s[0] = fma(w, bx, fma(-hd, dx, s[0]));
        s[1] = fma(w, by, fma(-hd, dy, s[1]));
        s[2] = fma(w, dd, s[2]);
        s[3] = fma(qy, fma(aix, dx, __dmul_rn(aiy, dy)), s[3]);
    }
}

template <int MODE, class Split>
__device__ __forceinline__ void adj_group_sums(const AdjCloud &d, int tile, const double *x, const double *y,
                                               const double *q, const double *ax, const double *ay, Split in,
                                               AdjGroupSmem<MODE == 0 ? 2 : 4> &sm) {
    constexpr int NS = MODE == 0 ? 2 : 4;
    cg::cluster_group cl = cg::this_cluster();
    const int S = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int li = 32 * tile + lane, n = d.n;
    const bool valid = li < n;
    double sum[NS];
#pragma unroll
    for (int k = 0; k < NS; k++) sum[k] = 0.0;
    if (d.flags & kShieldedCoulomb) {
        x += d.off;
        y += d.off;
        q += d.off;
        if (MODE == 1) ax += d.off, ay += d.off;
        auto pa = [&](int k) { return in(d.off + k); };
        float px2 = 0.0f, py2 = 0.0f, nu = INFINITY;
        double xi = 0.0, yi = 0.0, aix = 0.0, aiy = 0.0;
        if (valid) {
            const float4 A = pa(li);
            px2 = 2.0f * A.x;
            py2 = 2.0f * A.y;
            nu = A.w;
            xi = x[li];
            yi = y[li];
            if (MODE == 1) aix = ax[li], aiy = ay[li];
        }
        if (warp == 0) {
            sm.ix[lane] = xi;
            sm.iy[lane] = yi;
            if (MODE == 1) sm.iax[lane] = aix, sm.iay[lane] = aiy;
        }
        for (int k = tid; k < kExp2Size; k += 32 * kAdjWarps) sm.tab[k] = g_exp2_table.v[k];
        __syncthreads();
        HitWarp<HitResult<NS>> &W = sm.w[warp];
        const double *tab = sm.tab;
        const Yukawa64 K = d.y64;
        auto eval = [&](int il, int j) {
            HitResult<NS> r;
#pragma unroll
            for (int k = 0; k < NS; k++) r.v[k] = 0.0;
            const bool m1 = MODE == 1;
            adj_pair64<MODE>(K, tab, __dsub_rn(sm.ix[il], x[j]), __dsub_rn(sm.iy[il], y[j]), q[j],
                             m1 ? sm.iax[il] : 0.0, m1 ? sm.iay[il] : 0.0, m1 ? ax[j] : 0.0, m1 ? ay[j] : 0.0, true,
                             r.v);
            return r;
        };
        int nk = 0, hits = 0;
        for (int g = warp * S + rank; 32 * g < n; g += kAdjWarps * S) {
            const int h = hit_filter(W, nk, g, tile, pa, n, px2, py2, nu);
            if (__reduce_add_sync(0xffffffffu, h) >= 704) {  // >= 11/16 of the pairs: lane by lane
                __syncwarp();
                const uint32_t m = W.mask[nk][lane];
                const int jn = min(32, n - 32 * g);
                for (int u = 0; u < jn; u++) {
                    const int j = 32 * g + u;
                    const bool m1 = MODE == 1;
                    adj_pair64<MODE>(K, tab, __dsub_rn(xi, x[j]), __dsub_rn(yi, y[j]), q[j], aix, aiy,
                                     m1 ? ax[j] : 0.0, m1 ? ay[j] : 0.0, (m >> u) & 1u, sum);
                }
                continue;
            }
            hits += h;
            if (++nk == kHitGroups || __reduce_add_sync(0xffffffffu, hits) >= 7 * 32) {
                __syncwarp();
                hit_flush(W, nk, sum, eval);
                nk = hits = 0;
            }
        }
        __syncwarp();
        hit_flush(W, nk, sum, eval);
    }
#pragma unroll
    for (int k = 0; k < NS; k++) sm.acc[warp][k][lane] = sum[k];
    __syncthreads();
    if (warp < NS) {
        double t = 0.0;
#pragma unroll
        for (int w = 0; w < kAdjWarps; w++) t = __dadd_rn(t, sm.acc[w][warp][lane]);
        sm.red[warp][lane] = t;
    }
    if (S > 1) {
        cl.sync();
        if (rank == 0 && warp < NS) {
            double t = sm.red[warp][lane];
            for (int r = 1; r < S; r++) t = __dadd_rn(t, *cl.map_shared_rank(&sm.red[warp][lane], r));
            sm.red[warp][lane] = t;
        }
    }
    __syncthreads();
}

// C q_i (and -kappa for the last) times the sums of lane's particle.
template <int MODE>
__device__ __forceinline__ void adj_group_scaled(const AdjCloud &d, const AdjGroupSmem<MODE == 0 ? 2 : 4> &sm,
                                                 double coulomb, double qi, double (&S)[4]) {
    const int lane = threadIdx.x & 31;
    const double cq = __dmul_rn(coulomb, qi);
    S[2] = S[3] = 0.0;
#pragma unroll
    for (int k = 0; k < (MODE == 0 ? 2 : 3); k++) S[k] = __dmul_rn(cq, sm.red[k][lane]);
    if (MODE == 1) S[3] = __dmul_rn(__dmul_rn(-d.kappa, cq), sm.red[MODE == 1 ? 3 : 0][lane]);
}

static __global__ void __launch_bounds__(32 * kAdjWarps) adj_step_fp64(const AdjCloud *__restrict__ desc,
                                                                       const int2 *__restrict__ groups,
                                                                       const AdjStepIO io, double coulomb) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    AdjGroupSmem<2> &sm = *reinterpret_cast<AdjGroupSmem<2> *>(smem_raw);
    cg::cluster_group cl = cg::this_cluster();
    const int2 g = groups[blockIdx.x / cl.num_blocks()];
    const AdjCloud &d = desc[g.x];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    adj_group_sums<0>(d, g.y, io.x, io.y, io.q, nullptr, nullptr, AdjStoredSplit{io.in.p}, sm);
    const int li = 32 * g.y + lane, i = d.off + li;
    if (cl.block_rank() == 0) {
        const bool valid = li < d.n;
        if (valid) {
            double S[4];
            adj_group_scaled<0>(d, sm, coulomb, io.q[i], S);
            const double v = adj_step_component(d, io, i, warp, S[warp & 1]);
            if (warp < 2) sm.xch[warp][lane] = v;
        }
        __syncthreads();
        if (valid && warp == 0 && io.stage < 4) adj_store_split(io.out, i, sm.xch[0][lane], sm.xch[1][lane], d.rc2_up);
    }
    if (cl.num_blocks() > 1) cl.sync();  // the other blocks' sums stay readable until here
}

static __global__ void __launch_bounds__(32 * kAdjWarps) adj_vjp_fp64(const AdjCloud *__restrict__ desc,
                                                                      const int2 *__restrict__ groups,
                                                                      const AdjVjpIO V, double coulomb) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    AdjGroupSmem<4> &sm = *reinterpret_cast<AdjGroupSmem<4> *>(smem_raw);
    cg::cluster_group cl = cg::this_cluster();
    const int2 g = groups[blockIdx.x / cl.num_blocks()];
    const AdjCloud &d = desc[g.x];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    adj_group_sums<1>(d, g.y, V.x, V.y, V.q, V.ax, V.ay, AdjStoredSplit{V.in.p}, sm);
    const int li = 32 * g.y + lane, i = d.off + li;
    if (cl.block_rank() == 0 && li < d.n) {
        double S[4];
        adj_group_scaled<1>(d, sm, coulomb, V.q[i], S);
        const double dkn = adj_vjp_component(d, V, i, warp, S);
        if (V.stage > 1) {
            if (warp >= 2) (warp == 2 ? V.axn : V.ayn)[i] = adj_next_force_adjoint(V, i, dkn);
            else if (warp == 0) adj_store_split(V.out, i, V.xn[i], V.yn[i], d.rc2_up);
        }
    }
    if (cl.num_blocks() > 1) cl.sync();
}

// Forces (MODE 0) or their VJP (MODE 1) alone, FP64.
template <int MODE>
__global__ void __launch_bounds__(32 * kAdjWarps) adj_once_fp64(const AdjCloud *__restrict__ desc,
                                                                const int2 *__restrict__ groups, const AdjOnce A,
                                                                double coulomb) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    auto &sm = *reinterpret_cast<AdjGroupSmem<MODE == 0 ? 2 : 4> *>(smem_raw);
    cg::cluster_group cl = cg::this_cluster();
    const int2 g = groups[blockIdx.x / cl.num_blocks()];
    const AdjCloud &d = desc[g.x];
    adj_group_sums<MODE>(d, g.y, A.x, A.y, A.q, A.ax, A.ay, AdjFormedSplit{A.x, A.y, d.rc2_up}, sm);
    const int li = 32 * g.y + (int)(threadIdx.x & 31);
    if (cl.block_rank() == 0 && threadIdx.x < 32 && li < d.n) {
        double S[4];
        adj_group_scaled<MODE>(d, sm, coulomb, A.q[d.off + li], S);
        adj_once_outputs<MODE>(d, A, d.off + li, S);
    }
    if (cl.num_blocks() > 1) cl.sync();
}

}  // namespace dm
