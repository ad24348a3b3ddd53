// dm_api.cu -- host side of the C ABI declared in include/demon_gb300.h.
//
// One dm_ctx = one GPU + one stream.  One dm_cloud = one device-resident
// particle cloud (layout in dm_device.cuh).  Per RK4 step the library issues
// two passes of two force evaluations each (dm_pair.cuh); fixed-dt step
// sequences are captured once into a CUDA graph and replayed.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <utility>
#include <vector>

#include "../../include/demon_gb300.h"
#include "dm_misc.cuh"
#include "dm_pair.cuh"
#include "dm_sort.cuh"
#include "dm_batch.cuh"
#include "dm_adjoint.cuh"

using namespace dm;

static_assert(sizeof(dm_force_params) == sizeof(ForceParams), "force params layout");

namespace {

std::string g_create_error;

// FP64 clouds above this size are swept group by group within reach, which
// needs the Morton order; up to it every group pair is filtered and the cloud
// stays in whatever order it is in (at 4096 particles the filter of all 16,384
// group pairs costs ~3 us a stage, the re-sort ~18 us a step).
constexpr int kFp64UnsortedMax = 4096;
constexpr int kGraphSteps = 16;
// States of at most this many particles in pageable memory cross through the
// context's page-locked staging (64 bytes each) and a copy kernel; larger ones by
// DMA.  Eight pageable copies cost the host a fixed ~70 us a round trip (upload
// and download), staging ~2.3 us per 1024 particles, two passes of the host over
// the state: 1024 particles 71 us by DMA, 37 staged; 8192 87 and 59; 16,384 108
// and 86; 24,576 111 and 120; 65,536 129 and 302.
constexpr int kStagedCopyMax = 16384;

}  // namespace

struct dm_ctx {
    int device = 0;
    cudaStream_t own_stream = nullptr;
    cudaStream_t stream = nullptr;
    int num_sms = 0;
    std::string err;
    bool prof = false;
    bool autotune = true;
    long long launches = 0;  // kernels this library has launched on the context
    std::map<long long, std::pair<int, int>> tune_cache;  // (n, precision) -> (variant, split)
    std::vector<std::pair<cudaEvent_t, cudaEvent_t>> prof_events;
    size_t prof_used = 0;
    double prof_pairs = 0.0;
    long long prof_launches = 0;
    int *h_err = nullptr;  // pinned word for the device error flags (read with each download)
    double *h_stage = nullptr, *h_stage_dev = nullptr;  // page-locked [2][4][stage_n]: uploads, downloads
    int stage_n = 0;                                    // largest cloud it holds
    cudaEvent_t stage_read = nullptr;                   // the last staged upload has been read
    AdaptiveResult *h_adapt = nullptr;  // page-locked: the adaptive time step's result
    int sort_ctas = 0;     // blocks of the one-cluster sort (0: not chosen yet)

    int fail(int code, const char *fmt, ...) {
        char buf[512];
        va_list ap;
        va_start(ap, fmt);
        vsnprintf(buf, sizeof(buf), fmt, ap);
        va_end(ap);
        err = buf;
        return code;
    }
};

struct GraphKey {
    int precision;
    int nsteps;
    double dt;
    int slot;  // step counter / force time slot current at the first step
    bool operator<(const GraphKey &o) const {
        if (precision != o.precision) return precision < o.precision;
        if (nsteps != o.nsteps) return nsteps < o.nsteps;
        if (slot != o.slot) return slot < o.slot;
        return dt < o.dt;
    }
};

// A captured block of steps and the kernels in it.
struct StepGraph {
    cudaGraphExec_t exec;
    long long launches;
};

struct dm_cloud {
    dm_ctx *ctx = nullptr;
    int n = 0, n_pad = 0;
    void *block = nullptr;
    CloudDev d{};
    ForceParams f{};
    double coulomb = 0.0;
    double *d_fx = nullptr, *d_fy = nullptr;
    double *d_dt = nullptr;
    double *d_diag = nullptr;    // diagnostics: [kDiagBlocks][5] partial sums, then the 5 results
    unsigned int *d_min = nullptr;  // adaptive time step: least checked r^2, finished blocks
    int order = 4;               // integrator: 4 = Runge_Kutta4, 2 = Runge_Kutta2
    int eval_thermal_stage = 1;  // substep of the thermal kicks in force-only evaluations
    bool boxes_valid[4] = {false, false, false, false};  // group boxes (culling) match position set b
    bool supers_valid[2] = {false, false};  // super group boxes match sets 2 p, 2 p + 1
    bool mid_valid = false;      // position set 1 is the midpoint for time step mid_dt
    double mid_dt = 0.0;
    int slot = 0;                // current step counter / force time slot (RK2 steps alternate it)
    bool capturing = false;      // the running call is recorded by the caller's stream capture
    bool captured = false;       // some call was: replays change the state unseen
    bool split_stale = false;    // ... and may leave set 0's filter bounds of other force parameters
    int split[2] = {0, 0};  // cluster size per precision (0 = not chosen yet)
    int tuned_variant[2] = {-1, -1};  // per precision: index into kVariants
    float2 *partial = nullptr;         // [2 partial_cap][2][n_pad] non-cluster partial sums (per set and rank, axis)
    int partial_cap = 0;
    std::vector<void *> retired;       // outgrown partial-sum buffers that recorded steps may still use
    SortScratch sort{};
    int sort_blocks = 0;
    int reorder_interval = 1;   // steps between Morton re-sorts (0 = never)
    bool keep_orders = true;    // a due sort leaves an order that is still good (no interval was asked for)
    bool order_dirty = true;    // re-sort before the next step ...
    int dirty_upload = 0;       // ... if upload of this number changed the state (0: in any case)
    int uploads = 0;
    unsigned long long host_steps = 0;  // RK4 steps enqueued so far
    std::map<GraphKey, StepGraph> graphs;
    cudaStream_t graph_stream = nullptr;  // stream the graphs were built for

    void drop_graphs() {
        for (auto &kv : graphs) cudaGraphExecDestroy(kv.second.exec);
        graphs.clear();
    }
    // the state (set 0) was rewritten: what was derived from it is stale;
    // boxes: set 0's group boxes were rewritten with it
    void state_changed(bool boxes) {
        boxes_valid[0] = boxes;
        boxes_valid[1] = mid_valid = supers_valid[0] = false;
    }
    ~dm_cloud() {
        if (partial) cudaFree(partial);
        for (void *p : retired) cudaFree(p);
    }
};

#define DM_CUDA(ctx, call)                                                                   \
    do {                                                                                     \
        cudaError_t e_ = (call);                                                             \
        if (e_ != cudaSuccess)                                                               \
            return (ctx)->fail(DM_ERR_CUDA, "%s failed: %s (%s:%d)", #call,                 \
                               cudaGetErrorString(e_), __FILE__, __LINE__);                 \
    } while (0)

namespace {

size_t align256(size_t v) { return (v + 255) & ~(size_t)255; }

// Status for device error flags h already read back (and clears them).
int device_error_status(dm_ctx *ctx, dm_cloud *c, int h) {
    if (h) {
        DM_CUDA(ctx, cudaMemsetAsync(c->d.err, 0, sizeof(int), ctx->stream));
        if (h & 2) return ctx->fail(DM_ERR_NUMERIC, "zero particle separation in the adaptive time step test");
        if (h & kErrSortPermutation)
            return ctx->fail(DM_ERR_CUDA, "internal error: the Morton sort produced an invalid permutation");
        return ctx->fail(DM_ERR_NUMERIC, "non-finite particle position after a stage (error bits 0x%x)", h);
    }
    return DM_OK;
}

// The autotuners' weights of a candidate's time on the cloud as it is and on
// its dense copy: a confined cloud passes through its focus in about one step
// of four to seven.  (With equal weights the dense copy, five times as slow,
// decided alone: the batch of 256 clouds took a variant 0.7% better in the sum
// and 29% slower on the clouds at rest.)
constexpr float kTuneWeight[2] = {3.0f, 1.0f};

// DM_TUNE_VERBOSE: the autotuners' timings of every candidate on stderr.
bool tune_verbose() {
    const char *e = getenv("DM_TUNE_VERBOSE");
    return e && e[0] && e[0] != '0';
}

// The FP32C sweep's threshold for evaluating a filtered chunk directly
// (StageParams::direct_min): at least this many of a slot's 128 (lane, j)
// pairs passed the filter.  DM_DIRECT_MIN_HITS overrides it (1..129; 129
// never evaluates directly).
int direct_min_hits() {
    static const int v = [] {
        const char *e = getenv("DM_DIRECT_MIN_HITS");
        const int k = e ? atoi(e) : 0;
        return (k >= 1 && k <= 129) ? k : 48;
    }();
    return v;
}

// StageParams::near_direct_f2: groups whose farthest separation from the
// tile is within F = 1.6 r_c are evaluated without the filter (measured on
// disk16k: the collapsed-state launch 154.8 -> 146.0 us, the densest step
// -7%, calm steps +1%; 1.3-2.5 within 1% of each other).
// DM_NEAR_DIRECT_F overrides F (0 turns the class off; at most 4).
float near_direct_f2() {
    static const float v = [] {
        const char *e = getenv("DM_NEAR_DIRECT_F");
        double f = e ? atof(e) : 1.6;
        if (!(f >= 0.0 && f <= 4.0)) f = 0.0;
        return (float)(f * f);
    }();
    return v;
}

// kappa*log2(e) as a float pair (hi + lo to ~2^-48 relative).
void kappa_log2e(double kappa, float &hi, float &lo) {
    const double k = kappa * 1.4426950408889634;
    hi = (float)k;
    lo = (float)(k - (double)hi);
}

// The parameters of pass 0 or 1 of a step, or (mode kModeForceOnly) of one
// force evaluation at position set buf, evaluated nsets times.
StageParams make_stage_params(dm_cloud *c, int pass, int mode, double dt, const double *dt_dev, int buf = 0,
                              int nsets = 1) {
    StageParams P{};
    P.c = c->d;
    P.f = c->f;
    P.pass = pass;
    P.order = c->order;
    P.mode = mode;
    P.nsets = (mode == kModeForceOnly) ? nsets : 2;
    P.buf[0] = (mode == kModeForceOnly) ? buf : 2 * pass;
    P.buf[1] = (mode == kModeForceOnly) ? buf : 2 * pass + 1;
    P.slot = c->slot;
    P.therm_stage = c->eval_thermal_stage;
    P.dt = dt;
    P.dt_dev = dt_dev;
    P.coulomb = c->coulomb;
    P.fx_out = c->d_fx;
    P.fy_out = c->d_fy;
    const double kappa = c->f.shielding;
    P.rc2 = (kappa > 0.0) ? (10.0 / kappa) * (10.0 / kappa) : INFINITY;
    // FP32 r^2 is within ~6 ulp of the FP64 value; outside this band the
    // FP32 decision cannot differ from the reference's FP64 one
    P.rc2_lo = (float)(P.rc2 * (1.0 - 4e-6));
    P.rc2_hi = (float)(P.rc2 * (1.0 + 4e-6));
    P.kappa_f = (float)kappa;
    P.nkl2e = (float)(-kappa * 1.4426950408889634);
    P.y64 = make_yukawa64(kappa, P.rc2);
    P.direct_min = direct_min_hits();
    P.near_direct_f2 = near_direct_f2();
    return P;
}

// ---------------------------------------------------------------------------
// Kernel variants and the autotuner
// ---------------------------------------------------------------------------
struct Variant {
    const char *name;
    int precision;
    bool cluster;  // reduce through a thread-block cluster (else global partials + stage_finish)
    bool cull;     // skip j groups whose box is beyond the cutoff from the tile's (group_bounds first)
    int nt;        // threads per CTA (cluster variants: and position set)
    int tile;      // particles per i tile
    int min_j;     // j particles per block of a split at least
    size_t smem;   // cluster variants: for both position sets
    const void *fn;
    cudaError_t (*launch)(const cudaLaunchConfig_t *, const StageParams &);
};

template <int NW, int ILP, int TC, bool CL, bool CULL>
cudaError_t launch_fp32c(const cudaLaunchConfig_t *cfg, const StageParams &P) {
    return cudaLaunchKernelEx(cfg, pair_stage_fp32c<NW, ILP, TC, CL, CULL>, P);
}
template <int NW, bool CULL>
cudaError_t launch_fp64(const cudaLaunchConfig_t *cfg, const StageParams &P) {
    return cudaLaunchKernelEx(cfg, pair_group_fp64<NW, CULL>, P);
}

#define DM_FP32C_VARIANT(NW, ILP, TC, CL)                                                        \
    {"fp32c<" #NW "," #ILP "," #TC "," #CL ">", DM_FP32C, CL, false, NW * 32, 32 * ILP, 64 * NW, \
     (CL ? 2 : 1) * Fp32cSmem<NW, ILP, TC>::bytes, (const void *)pair_stage_fp32c<NW, ILP, TC, CL, false>,       \
     launch_fp32c<NW, ILP, TC, CL, false>}
#define DM_FP32C_CULL_VARIANT(NW, ILP, TC, CL)                                                   \
    {"fp32c<" #NW "," #ILP "," #TC "," #CL ",cull>", DM_FP32C, CL, true, NW * 32, 32 * ILP, 64 * NW, \
     (CL ? 2 : 1) * Fp32cSmem<NW, ILP, TC>::bytes, (const void *)pair_stage_fp32c<NW, ILP, TC, CL, true>,        \
     launch_fp32c<NW, ILP, TC, CL, true>}

#define DM_FP64_VARIANT(NW, CULL, SUFFIX)                                                        \
    {"fp64<" #NW SUFFIX ">", DM_FP64, true, CULL, NW * 32, 32, 32 * NW, sizeof(Group64Smem<NW>), \
     (const void *)pair_group_fp64<NW, CULL>, launch_fp64<NW, CULL>}

const Variant kVariants[] = {
    DM_FP32C_VARIANT(8, 4, 256, true),
    DM_FP32C_VARIANT(8, 4, 256, false),
    DM_FP32C_VARIANT(4, 4, 256, true),
    DM_FP32C_VARIANT(4, 4, 256, false),
    DM_FP32C_VARIANT(16, 4, 256, false),
    DM_FP32C_VARIANT(8, 2, 256, false),
    DM_FP32C_CULL_VARIANT(8, 4, 256, false),
    DM_FP32C_CULL_VARIANT(4, 4, 256, false),
    DM_FP32C_CULL_VARIANT(8, 2, 256, false),
    DM_FP32C_CULL_VARIANT(4, 2, 128, false),
    DM_FP32C_CULL_VARIANT(8, 4, 256, true),
    DM_FP64_VARIANT(8, false, ""),
    DM_FP64_VARIANT(8, true, ",near"),
    DM_FP64_VARIANT(4, true, ",near"),
    DM_FP64_VARIANT(4, false, ""),
};
constexpr int kNumVariants = (int)(sizeof(kVariants) / sizeof(kVariants[0]));
constexpr int kDefaultVariant32 = 0;
constexpr int kDefaultVariant64 = kNumVariants - 1, kDefaultVariant64Cull = kNumVariants - 2;
constexpr int kMaxSplitGlobal = 64;
constexpr int kMaxSplitCluster = 16;
constexpr int kSuperMin = 1024;      // 32-particle groups from which super group boxes are kept

int ensure_kernel_attrs(dm_ctx *ctx) {
    static bool done[64] = {false};
    int dev = ctx->device;
    if (dev < 0 || dev >= 64) dev = 0;
    if (done[dev]) return DM_OK;
    for (int v = 0; v < kNumVariants; v++) {
        const Variant &k = kVariants[v];
        if (k.cluster)
            DM_CUDA(ctx, cudaFuncSetAttribute(k.fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        DM_CUDA(ctx, cudaFuncSetAttribute(k.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)k.smem));
    }
    DM_CUDA(ctx, cudaFuncSetAttribute(sort_cluster<8>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)sort_cluster_smem<8>()));
    DM_CUDA(ctx, cudaFuncSetAttribute(sort_cluster<16>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    DM_CUDA(ctx, cudaFuncSetAttribute(sort_cluster<16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)sort_cluster_smem<16>()));
    done[dev] = true;
    return DM_OK;
}

template <int CTAS>
cudaLaunchConfig_t sort_cluster_cfg(cudaStream_t s, cudaLaunchAttribute *attr) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(CTAS);
    cfg.blockDim = dim3(kSortClusterThreads);
    cfg.dynamicSmemBytes = sort_cluster_smem<CTAS>();
    cfg.stream = s;
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = CTAS;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cfg;
}

// Blocks of the one-cluster sort on this device: 16 (half the elements per
// SM of 8) when a 16-block cluster of it can be scheduled, else 8;
// DM_SORT_CLUSTER_CTAS=8 keeps 8.
int choose_sort_ctas(dm_ctx *ctx) {
    if (ctx->sort_ctas) return DM_OK;
    int rc = ensure_kernel_attrs(ctx);
    if (rc) return rc;
    const char *e = getenv("DM_SORT_CLUSTER_CTAS");
    int ctas = (e && atoi(e) == 8) ? 8 : 16;
    if (ctas == 16) {
        cudaLaunchAttribute attr[2];
        cudaLaunchConfig_t cfg = sort_cluster_cfg<16>(ctx->stream, attr);
        int nc = 0;
        if (cudaOccupancyMaxActiveClusters(&nc, sort_cluster<16>, &cfg) != cudaSuccess || nc < 1) {
            cudaGetLastError();
            ctas = 8;
        }
    }
    ctx->sort_ctas = ctas;
    return DM_OK;
}

// Launch of a kernel that starts with pdl_wait(): it may be scheduled while
// the previous kernel in the stream finishes.
template <typename... KArgs, typename... Args>
cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                       Args &&...args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

// Whether steps and force evaluations of n particles run on the Morton order.
bool wants_order(int n, int precision) { return precision == DM_FP32C || n > kFp64UnsortedMax; }

// attr must hold 2 entries: programmatic serialization (see pdl_wait) and,
// for cluster variants, the cluster shape.
cudaLaunchConfig_t make_cfg(dm_ctx *ctx, const Variant &k, int ntiles, int S, int nsets, cudaLaunchAttribute *attr) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ntiles * S * (k.cluster ? 1 : nsets), 1, 1);
    cfg.blockDim = dim3(k.nt * (k.cluster ? nsets : 1), 1, 1);
    cfg.dynamicSmemBytes = k.smem;
    cfg.stream = ctx->stream;
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (k.cluster) {
        attr[1].id = cudaLaunchAttributeClusterDimension;
        attr[1].val.clusterDim.x = S;
        attr[1].val.clusterDim.y = 1;
        attr[1].val.clusterDim.z = 1;
        cfg.numAttrs = 2;
    }
    return cfg;
}

// j split S for a variant from a cost model: all CTAs do equal work (1/S of a
// tile), so a launch takes as long as its busiest SM.  With X co-resident
// clusters (or CTAs) the tiles run in ceil(ntiles / X) waves and within a
// wave the busiest SM holds ceil(CTAs_in_wave / num_sms) CTAs.  Cost = sum
// over waves of that count / S; on ties (within 2%) the larger S wins, since
// more co-resident CTAs hide latency better.
int model_split(dm_ctx *ctx, const Variant &k, int n, int n_pad) {
    const int ntiles = (n + k.tile - 1) / k.tile;
    const int smax = k.cluster ? kMaxSplitCluster : kMaxSplitGlobal;
    int best_s = 1;
    double best_cost = 1e300;
    for (int S = 1; S <= smax; S++) {
        if (S > 1 && n_pad / S < k.min_j) break;
        int slots = 0;
        if (k.cluster) {
            cudaLaunchAttribute attr[2];
            cudaLaunchConfig_t cfg = make_cfg(ctx, k, ntiles, S, 2, attr);
            if (cudaOccupancyMaxActiveClusters(&slots, k.fn, &cfg) != cudaSuccess) {
                cudaGetLastError();
                continue;
            }
        } else {
            int per_sm = 0;
            if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k.fn, k.nt, k.smem) != cudaSuccess) {
                cudaGetLastError();
                continue;
            }
            slots = per_sm * ctx->num_sms / (2 * S);  // co-resident tiles (both position sets)
        }
        if (slots <= 0) continue;
        double cost = 0.0;
        for (int left = ntiles; left > 0; left -= slots) {
            const int in_wave = std::min(left, slots) * S * (k.cluster ? 1 : 2);
            cost += (double)((in_wave + ctx->num_sms - 1) / ctx->num_sms) / S;
        }
        if (cost <= best_cost * 1.02) {
            best_cost = std::min(best_cost, cost);
            best_s = S;
        }
    }
    return best_s;
}

int ensure_partial(dm_cloud *c, int S) {
    if (S <= c->partial_cap) return DM_OK;
    dm_ctx *ctx = c->ctx;
    DM_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (c->partial && c->captured) c->retired.push_back(c->partial);  // the caller's graphs hold its address
    else if (c->partial) cudaFree(c->partial);
    c->partial = nullptr;
    c->partial_cap = 0;
    cudaError_t e = cudaMalloc((void **)&c->partial, (size_t)S * 4 * c->n_pad * sizeof(float2));
    if (e != cudaSuccess)
        return ctx->fail(DM_ERR_NOMEM, "partial-sum buffer (%d x %d): %s", S, c->n_pad, cudaGetErrorString(e));
    c->partial_cap = S;
    c->drop_graphs();
    return DM_OK;
}

// One pass: the pair kernel (+ stage_finish for non-cluster variants), after
// the group boxes that it needs and lacks.
int launch_variant(dm_cloud *c, int vi, int S, StageParams P) {
    dm_ctx *ctx = c->ctx;
    const Variant &k = kVariants[vi];
    P.split = S;
    P.partial = c->partial;
    const int ngroups = (c->n + 31) / 32;
    if (c->split_stale) {
        init_positions<<<(c->n_pad + 255) / 256, 256, 0, ctx->stream>>>(c->d);
        DM_CUDA(ctx, cudaGetLastError());
        ctx->launches++;
        c->split_stale = false;
    }
    cudaLaunchAttribute attr[2];
    cudaLaunchConfig_t cfg = make_cfg(ctx, k, (c->n + k.tile - 1) / k.tile, S, P.nsets, attr);
    if (k.cull) {
        for (int e = 0; e < P.nsets; e++) {
            const int b = P.buf[e];
            if (c->boxes_valid[b]) continue;
            DM_CUDA(ctx, launch_pdl(group_bounds, dim3((c->n_pad + 255) / 256), dim3(256), 0, ctx->stream, c->d, b));
            ctx->launches++;
            c->boxes_valid[b] = true;
            c->supers_valid[b / 2] = false;
        }
        if (c->d.gsuper[0] && !c->supers_valid[P.buf[0] / 2]) {
            const int nsuper = (ngroups + 31) / 32;
            DM_CUDA(ctx, launch_pdl(super_bounds, dim3((2 * nsuper + 7) / 8), dim3(256), 0, ctx->stream, c->d,
                                    P.buf[0] & 2, ngroups));
            ctx->launches++;
            c->supers_valid[P.buf[0] / 2] = true;
        }
    }
    // profiling (dm_ctx_profile_enable): CUDA events around the pair launch
    // alone (a cluster variant's launch includes its epilogue)
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    if (ctx->prof) {
        if (ctx->prof_used == ctx->prof_events.size()) {
            cudaEvent_t a, b;
            DM_CUDA(ctx, cudaEventCreate(&a));
            DM_CUDA(ctx, cudaEventCreate(&b));
            ctx->prof_events.push_back({a, b});
        }
        e0 = ctx->prof_events[ctx->prof_used].first;
        e1 = ctx->prof_events[ctx->prof_used].second;
        ctx->prof_used++;
        DM_CUDA(ctx, cudaEventRecord(e0, ctx->stream));
    }
    DM_CUDA(ctx, k.launch(&cfg, P));
    ctx->launches++;
    if (ctx->prof) {
        DM_CUDA(ctx, cudaEventRecord(e1, ctx->stream));
        ctx->prof_launches++;
        ctx->prof_pairs += (double)P.nsets * (double)c->n * (double)(c->n - 1);
    }
    if (!k.cluster) {
        if (P.f.flags & ~kBasicForces)
            DM_CUDA(ctx, launch_pdl(stage_finish<true>, dim3(ngroups), dim3(64 * kTermParts), 0, ctx->stream, P));
        else
            DM_CUDA(ctx, launch_pdl(stage_finish<false>, dim3(ngroups), dim3(128), 0, ctx->stream, P));
        ctx->launches++;
    }
    if (P.mode == kModeForceOnly) return DM_OK;
    // the epilogue leaves two position sets with their boxes
    const int ob = (P.pass == 0) ? 2 : 0;
    c->boxes_valid[ob] = c->boxes_valid[ob + 1] = true;
    c->supers_valid[ob / 2] = false;
    if (P.order == 2) {
        if (c->captured) {
            DM_CUDA(ctx, launch_pdl(adopt_sets, dim3((c->n + 255) / 256), dim3(256), 0, ctx->stream, c->d, ngroups));
            ctx->launches++;
        } else {
            swap_sets(c->d);
        }
        c->boxes_valid[0] = c->boxes_valid[1] = true;
        c->supers_valid[0] = false;
    }
    if (P.order == 2 || P.pass == 1) {  // the step is done: set 1 is the next step's midpoint for the same dt
        c->mid_valid = P.dt_dev == nullptr;
        c->mid_dt = P.dt;
        if (P.order == 2) c->slot ^= 1;
    }
    return DM_OK;
}

int tune_precision(dm_cloud *c, int precision);
int reorder(dm_cloud *c, double dt = 0.0, bool mid = false, bool force = true);

int ensure_tuned(dm_cloud *c, int precision) {
    const int rc = ensure_kernel_attrs(c->ctx);
    if (rc) return rc;
    return (c->tuned_variant[precision == DM_FP32C ? 1 : 0] < 0) ? tune_precision(c, precision) : DM_OK;
}

// One pass (or force evaluation) with the cloud's tuned variant and split.
int launch_tuned(dm_cloud *c, int precision, const StageParams &P) {
    const int pi = precision == DM_FP32C ? 1 : 0;
    return launch_variant(c, c->tuned_variant[pi], c->split[pi], P);
}

// The passes of one step from set 0 (and set 1, if it is the midpoint for
// this dt; dt_dev: the adaptive dt, never).
int launch_step(dm_cloud *c, int precision, double dt, const double *dt_dev) {
    dm_ctx *ctx = c->ctx;
    int rc = ensure_tuned(c, precision);  // may use set 1
    if (rc) return rc;
    if (dt_dev || !c->mid_valid || c->mid_dt != dt) {
        DM_CUDA(ctx, launch_pdl(prepare_midpoint, dim3((c->n + 255) / 256), dim3(256), 0, ctx->stream, c->d, dt,
                                dt_dev));
        ctx->launches++;
        c->boxes_valid[1] = true;
        c->supers_valid[0] = false;
        c->mid_valid = dt_dev == nullptr;
        c->mid_dt = dt;
    }
    for (int pass = 0; pass < c->order / 2 && !rc; pass++)
        rc = launch_tuned(c, precision, make_stage_params(c, pass, kModeStep, dt, dt_dev));
    return rc;
}

// Autotuner: times every variant of this precision over a set of splits on
// THIS cloud (force-only launches: no state changes), keeps the fastest.
// Results are cached per (precision, n) in the context.  When disabled, the
// default variant and the cost-model split are used.
int tune_precision(dm_cloud *c, int precision) {
    dm_ctx *ctx = c->ctx;
    const int pi = precision == DM_FP32C ? 1 : 0;
    const long long key = ((long long)c->n << 1) | pi;
    auto hit = ctx->tune_cache.find(key);
    if (hit != ctx->tune_cache.end()) {
        c->tuned_variant[pi] = hit->second.first;
        c->split[pi] = hit->second.second;
        if (!kVariants[c->tuned_variant[pi]].cluster) return ensure_partial(c, c->split[pi]);
        return DM_OK;
    }
    const bool order = wants_order(c->n, precision);
    const int defv = precision == DM_FP32C ? kDefaultVariant32 : order ? kDefaultVariant64Cull : kDefaultVariant64;
    int best_v = defv, best_s = model_split(ctx, kVariants[defv], c->n, c->n_pad);
    if (ctx->autotune) {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        DM_CUDA(ctx, cudaStreamIsCapturing(ctx->stream, &cs));
        if (cs != cudaStreamCaptureStatusNone)
            return ctx->fail(DM_ERR_STATE, "autotuning needs an uncaptured stream (run one step first)");
        if (order && c->order_dirty) {  // tune on the particle order the steps will see
            int rc = reorder(c);
            if (rc) return rc;
        }
        // Time every candidate on two states: the cloud as it is (buffer 0)
        // and, unless it is dense already, a copy squeezed about its centre
        // so that ~30% of the pairs are inside the cutoff (buffer 1).  A
        // trajectory passes through both kinds (a confined cloud collapses
        // and re-expands), and the best shape differs between them.
        const bool big = (double)c->n * c->n > 4e9;  // ~64k particles: keep tuning short
        int nstates = 1;
        // FP64: the cloud as it is decides -- dense copies are FP64-pipe bound
        // whatever the split (within 16% of each other at 16,384 particles,
        // where the cloud at rest takes 45 to 250 us).
        if (!big && precision == DM_FP32C && !c->order_dirty && c->d.rc2 > 0.0 && std::isfinite(c->d.rc2)) {
            double v[4];  // bounding box min x, min y, max x, max y
            DM_CUDA(ctx, cudaMemcpyAsync(v, c->sort.box + 4, sizeof v, cudaMemcpyDeviceToHost, ctx->stream));
            DM_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
            const double half = 0.5 * std::max(v[2] - v[0], v[3] - v[1]);
            const double lam = 1.8 * std::sqrt(c->d.rc2) / half;
            if (std::isfinite(half) && half > 0.0 && lam < 0.9) {
                c->boxes_valid[1] = c->mid_valid = c->supers_valid[0] = false;
                tune_compress<<<(c->n + 255) / 256, 256, 0, ctx->stream>>>(c->d, 0.5 * (v[0] + v[2]),
                                                                            0.5 * (v[1] + v[3]), lam);
                DM_CUDA(ctx, cudaGetLastError());
                nstates = 2;
            }
        }
        cudaEvent_t a, b;
        DM_CUDA(ctx, cudaEventCreate(&a));
        DM_CUDA(ctx, cudaEventCreate(&b));
        float best_ms = 1e30f;
        const bool verbose = tune_verbose();
        // culling variants first: most of the others are dropped after one
        // launch (a candidate whose first launch alone costs more than 1.3
        // times the best total is not timed further)
        std::vector<int> candidates;
        for (const bool cull : {true, false})
            for (int vi = 0; vi < kNumVariants; vi++)
                if (kVariants[vi].cull == cull) candidates.push_back(vi);
        for (const int vi : candidates) {
            const Variant &k = kVariants[vi];
            if (k.precision != precision || (precision == DM_FP64 && k.cull != order)) continue;
            const int sm = model_split(ctx, k, c->n, c->n_pad);
            std::vector<int> cands = {sm};
            if (big && !k.cluster && k.cull) cands = {1, 2, 4};
            const int extra_c[] = {1, 2, 3, 4, 6, 8, 16};
            const int extra_g[] = {1, 2, 3, 4, 5, 6, 8, 12, 16, 24, 32};
            if (!big) {
                if (k.cluster) cands.insert(cands.end(), std::begin(extra_c), std::end(extra_c));
                else cands.insert(cands.end(), std::begin(extra_g), std::end(extra_g));
            }
            std::sort(cands.begin(), cands.end());
            cands.erase(std::unique(cands.begin(), cands.end()), cands.end());
            for (int S : cands) {
                if (S > 1 && c->n_pad / S < k.min_j) continue;
                if (S > 1 && k.cull && 32 * S > c->n_pad) continue;  // j is dealt in groups of 32: idle ranks
                if (k.cluster) {
                    int nc = 0;
                    cudaLaunchAttribute attr[2];
                    cudaLaunchConfig_t cfg = make_cfg(ctx, k, (c->n + k.tile - 1) / k.tile, S, 2, attr);
                    if (cudaOccupancyMaxActiveClusters(&nc, k.fn, &cfg) != cudaSuccess || nc <= 0) {
                        cudaGetLastError();
                        continue;
                    }
                } else {
                    int rc = ensure_partial(c, S);
                    if (rc) return rc;
                }
                const int reps = big ? 1 : 3;
                float ms = 0.0f, ms_state[2] = {0.0f, 0.0f};
                for (int st = 0; st < nstates && ms < 1.3f * best_ms; st++) {
                    // both sets on the same buffer: a pass's work
                    const StageParams P = make_stage_params(c, 0, kModeForceOnly, 0.0, nullptr, st, 2);
                    // one launch, then the timed ones.  (Without a look at the first, which
                    // saves a synchronisation a candidate but times every poor one in
                    // full, tuning took 2.9 ms instead of 2.2 at 512 particles, 29
                    // instead of 19 at 4095; 151 particles 1.6 either way.)
                    for (int runs : {1, reps}) {
                        int rc = cudaEventRecord(a, ctx->stream) == cudaSuccess ? DM_OK : DM_ERR_CUDA;
                        for (int r = 0; r < runs && !rc; r++) rc = launch_variant(c, vi, S, P);
                        if (!rc) rc = cudaEventRecord(b, ctx->stream) == cudaSuccess ? DM_OK : DM_ERR_CUDA;
                        if (!rc) rc = cudaEventSynchronize(b) == cudaSuccess ? DM_OK : DM_ERR_CUDA;
                        if (rc) return rc == DM_ERR_CUDA ? ctx->fail(rc, "autotuner timing failed") : rc;
                        float one = 0.0f;
                        DM_CUDA(ctx, cudaEventElapsedTime(&one, a, b));
                        ms_state[st] = one / runs;
                        if (ms + kTuneWeight[st] * ms_state[st] >= 1.3f * best_ms) break;
                    }
                    ms += kTuneWeight[st] * ms_state[st];
                }
                if (verbose)
                    fprintf(stderr, "dm autotune n=%d %s split %d: %.4f ms (state) %.4f ms (dense copy)\n", c->n,
                            k.name, S, ms_state[0], ms_state[1]);
                if (ms < best_ms) {
                    best_ms = ms;
                    best_v = vi;
                    best_s = S;
                }
            }
        }
        cudaEventDestroy(a);
        cudaEventDestroy(b);
    }
    c->tuned_variant[pi] = best_v;
    c->split[pi] = best_s;
    ctx->tune_cache[key] = {best_v, best_s};
    if (!kVariants[best_v].cluster) return ensure_partial(c, best_s);
    return DM_OK;
}

// The radix passes over `bits` of z.keys[0] / z.vals[0] (`first`: the first
// digit's histogram is there); *cur: the buffer that holds the result.
int radix_passes(dm_ctx *ctx, const SortScratch &z, int n, int nblocks, int bits, bool first, const int *keep,
                 int *cur) {
    cudaStream_t s = ctx->stream;
    *cur = 0;
    for (int shift = 0; shift < bits; shift += kSortDigitBits) {
        if (shift > 0 || !first) {
            DM_CUDA(ctx, launch_pdl(radix_hist, dim3(nblocks), dim3(kSortThreads), 0, s,
                                    (const uint32_t *)z.keys[*cur], n, shift, z.hist, keep));
            ctx->launches++;
        }
        DM_CUDA(ctx, launch_pdl(radix_scan, dim3(kSortBuckets), dim3(256), 0, s, z.hist, nblocks, keep));
        DM_CUDA(ctx, launch_pdl(radix_scatter, dim3(nblocks), dim3(kSortThreads), 0, s,
                                (const uint32_t *)z.keys[*cur], (const int *)z.vals[*cur], z.keys[*cur ^ 1],
                                z.vals[*cur ^ 1], n, shift, (const uint32_t *)z.hist, keep));
        ctx->launches += 2;
        *cur ^= 1;
    }
    return DM_OK;
}

// Puts the cloud in Morton order (dm_sort.cuh); graph-capturable.  mid: the
// next step's time step is dt: the sort leaves its midpoint too.  Without
// `force` a cloud whose order is still good stays as it is.
int reorder(dm_cloud *c, double dt, bool mid, bool force) {
    dm_ctx *ctx = c->ctx;
    cudaStream_t s = ctx->stream;
    const int n = c->n;
    const int grid = (n + 255) / 256;
    SortScratch &z = c->sort;
    int cur = 0;
    if (n <= kSmallSortMax) {  // one cluster launch sorts and rewrites the cloud in place
        int rc = choose_sort_ctas(ctx);
        if (rc) return rc;
        cudaLaunchAttribute attr[2];
        const float4 *pa0 = c->d.pa[0];
        const bool mid_ready = c->mid_valid && c->mid_dt == dt && c->boxes_valid[1];
        force = force || !c->boxes_valid[0];
        const int upload = c->order_dirty ? c->dirty_upload : 0;
        if (ctx->sort_ctas == 16) {
            const cudaLaunchConfig_t cfg = sort_cluster_cfg<16>(s, attr);
            DM_CUDA(ctx, cudaLaunchKernelEx(&cfg, sort_cluster<16>, pa0, c->d, z, dt, mid, mid_ready, force, c->slot,
                                            upload));
        } else {
            const cudaLaunchConfig_t cfg = sort_cluster_cfg<8>(s, attr);
            DM_CUDA(ctx, cudaLaunchKernelEx(&cfg, sort_cluster<8>, pa0, c->d, z, dt, mid, mid_ready, force, c->slot,
                                            upload));
        }
        c->state_changed(true);
        c->boxes_valid[1] = c->mid_valid = mid;
        c->mid_dt = dt;
        c->split_stale = false;  // (stale: the sort was a forced one, which rewrites set 0)
        DM_CUDA(ctx, cudaGetLastError());
        ctx->launches += 1;
        c->order_dirty = false;
        return DM_OK;
    }
    const int nb = c->sort_blocks, cblocks = (c->n_pad + 255) / 256;
    const int mblocks = std::min(nb, kMomentBlocks);
    const float4 *pa0 = c->d.pa[0];
    const bool mid_ready = c->mid_valid && c->mid_dt == dt && c->boxes_valid[1];
    const int *keep = (force || !c->boxes_valid[0]) ? nullptr : z.keep;
    if (keep) {
        DM_CUDA(ctx, launch_pdl(order_check, dim3(1), dim3(1024), 0, s, c->d, z, c->slot,
                                c->order_dirty ? c->dirty_upload : 0));
        ctx->launches++;
    }
    DM_CUDA(ctx, launch_pdl(sort_moments, dim3(mblocks), dim3(256), 0, s, pa0, n, z.moments, keep));
    DM_CUDA(ctx, launch_pdl(sort_keys, dim3(nb), dim3(kSortThreads), 0, s, pa0, n, mblocks, z, keep));
    int rc = radix_passes(ctx, z, n, nb, kSortBits, true, keep, &cur);
    if (rc) return rc;
    DM_CUDA(ctx, launch_pdl(permute_gather, dim3(grid), dim3(256), 0, s, c->d, (const int *)z.vals[cur], z, keep));
    DM_CUDA(ctx, launch_pdl(permute_commit, dim3(cblocks), dim3(256), 0, s, c->d, z, dt, mid, mid_ready, keep));
    DM_CUDA(ctx, launch_pdl(order_record, dim3(1), dim3(1024), 0, s, c->d, z, c->slot, keep));
    ctx->launches++;
    c->state_changed(true);
    c->boxes_valid[1] = c->mid_valid = mid;
    c->mid_dt = dt;
    c->split_stale = false;
    ctx->launches += 4;
    c->order_dirty = false;
    return DM_OK;
}

// The re-sort at the start of a step, where one is due.
int reorder_if_due(dm_cloud *c, int precision, double dt, bool mid) {
    if (!wants_order(c->n, precision)) return DM_OK;
    if (c->order_dirty || (c->reorder_interval > 0 && c->host_steps % (unsigned)c->reorder_interval == 0))
        return reorder(c, dt, mid, (c->order_dirty && c->dirty_upload == 0) || !c->keep_orders);
    return DM_OK;
}

int enqueue_steps(dm_cloud *c, int nsteps, double dt, int precision) {
    for (int s = 0; s < nsteps; s++) {
        int rc = reorder_if_due(c, precision, dt, true);
        if (rc) return rc;
        rc = launch_step(c, precision, dt, nullptr);
        if (rc) return rc;
        c->host_steps++;
    }
    return DM_OK;
}

int run_steps(dm_cloud *c, int nsteps, double dt, int precision) {
    dm_ctx *ctx = c->ctx;
    if (ctx->prof || c->capturing || nsteps < kGraphSteps) return enqueue_steps(c, nsteps, dt, precision);
    if (c->graph_stream != ctx->stream) {
        c->drop_graphs();
        c->graph_stream = ctx->stream;
    }
    // the captured step sequence re-sorts at fixed positions: align the
    // host step counter and clear a pending re-sort first
    while (nsteps > 0 && wants_order(c->n, precision) &&
           (c->order_dirty || (c->reorder_interval > 0 && c->host_steps % kGraphSteps != 0))) {
        int rc = enqueue_steps(c, 1, dt, precision);
        if (rc) return rc;
        nsteps--;
    }
    if (nsteps < kGraphSteps) return enqueue_steps(c, nsteps, dt, precision);
    // the captured steps start from a midpoint left by the step before (or by
    // the re-sort that begins them, which may leave the order, and so needs
    // valid boxes, but always writes the midpoint): make it so, outside the capture
    int rc0 = ensure_tuned(c, precision);
    if (rc0) return rc0;
    const bool sorts = wants_order(c->n, precision) && c->reorder_interval > 0;
    if (sorts ? !c->boxes_valid[0] : !(c->mid_valid && c->mid_dt == dt)) {
        rc0 = enqueue_steps(c, 1, dt, precision);
        if (rc0) return rc0;
        return run_steps(c, nsteps - 1, dt, precision);
    }
    const GraphKey key{precision, kGraphSteps, dt, c->slot};
    auto it = c->graphs.find(key);
    if (it == c->graphs.end()) {
        cudaGraph_t g = nullptr;
        const unsigned long long saved = c->host_steps;
        const long long saved_launches = ctx->launches;
        // a replay meets particles that the block before it has moved: the
        // block forms the super group boxes it reads (set 0's may be valid now,
        // after a force evaluation)
        c->supers_valid[0] = c->supers_valid[1] = false;
        if (sorts) c->mid_valid = false;
        const CloudDev state = c->d;
        const int slot = c->slot;
        DM_CUDA(ctx, cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
        int rc = enqueue_steps(c, kGraphSteps, dt, precision);
        cudaError_t ec = cudaStreamEndCapture(ctx->stream, &g);
        c->host_steps = saved;  // capture recorded the steps, it did not run them
        const long long launches = ctx->launches - saved_launches;
        ctx->launches = saved_launches;
        if (rc || ec != cudaSuccess) {  // nothing has run: the state is where it was
            c->d = state;
            c->slot = slot;
            c->state_changed(false);
        }
        if (rc) {
            if (g) cudaGraphDestroy(g);
            return rc;
        }
        if (ec != cudaSuccess) return ctx->fail(DM_ERR_CUDA, "graph capture failed: %s", cudaGetErrorString(ec));
        cudaGraphExec_t ge = nullptr;
        ec = cudaGraphInstantiate(&ge, g, 0);
        cudaGraphDestroy(g);
        if (ec != cudaSuccess) return ctx->fail(DM_ERR_CUDA, "graph instantiate failed: %s", cudaGetErrorString(ec));
        it = c->graphs.emplace(key, StepGraph{ge, launches}).first;
    }
    const int reps = nsteps / kGraphSteps;
    for (int r = 0; r < reps; r++) {
        DM_CUDA(ctx, cudaGraphLaunch(it->second.exec, ctx->stream));
        c->host_steps += kGraphSteps;
        ctx->launches += it->second.launches;
        c->mid_valid = true;  // the replayed steps leave every position set's boxes and the midpoint
        c->mid_dt = dt;
        for (bool &v : c->boxes_valid) v = true;
        c->supers_valid[0] = false;
    }
    return enqueue_steps(c, nsteps - reps * kGraphSteps, dt, precision);
}

// What a caller's buffer is.  view: the device's own address of it when the
// device may dereference it (page-locked host memory: cudaHostAlloc,
// cudaMallocHost, cudaHostRegister, torch's pin_memory): on GB300 such buffers
// are read and written over NVLink-C2C by the copy kernel, one launch for all
// four arrays.  pageable: plain memory (or no buffer at all), which the host
// may read and write at once.  Page-locked, managed and device memory may be in
// use by work queued on the stream: copies of it stay in stream order.
struct Buffer {
    const void *view = nullptr;
    bool pageable = true;
    explicit Buffer(const void *p) {
        cudaPointerAttributes a;
        if (!p) return;
        pageable = false;
        if (cudaPointerGetAttributes(&a, p) != cudaSuccess) cudaGetLastError();
        else if (a.type == cudaMemoryTypeHost) view = a.devicePointer;
        else pageable = a.type == cudaMemoryTypeUnregistered;
    }
};
// The four arrays of a state.
struct StateBuffers {
    Buffer b[4];
    StateBuffers(const void *x, const void *y, const void *vx, const void *vy)
        : b{Buffer(x), Buffer(y), Buffer(vx), Buffer(vy)} {}
    bool viewed() const { return b[0].view && b[1].view && b[2].view && b[3].view; }
    bool pageable() const { return b[0].pageable && b[1].pageable && b[2].pageable && b[3].pageable; }
    double *view(int k) const { return (double *)b[k].view; }
};

// Whether a state of n particles is staged (see kStagedCopyMax); not under
// stream capture, where a replay has to read the caller's memory again.
bool staged_copies(dm_ctx *ctx, int n, const StateBuffers &B) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (!B.pageable()) return false;
    if (n > kStagedCopyMax || cudaStreamIsCapturing(ctx->stream, &cs) != cudaSuccess ||
        cs != cudaStreamCaptureStatusNone) {
        cudaGetLastError();
        return false;
    }
    if (n <= ctx->stage_n) return true;
    // for the cloud at hand: 1 MiB takes ~120 us to allocate, 32 KiB ~10
    int cap = 512;
    while (cap < n) cap *= 2;
    if (!ctx->stage_read && cudaEventCreateWithFlags(&ctx->stage_read, cudaEventDisableTiming) != cudaSuccess)
        ctx->stage_read = nullptr;
    void *h = nullptr, *d = nullptr;
    if (ctx->stage_read && cudaEventSynchronize(ctx->stage_read) == cudaSuccess &&
        cudaMallocHost(&h, 8 * (size_t)cap * sizeof(double)) == cudaSuccess &&
        cudaHostGetDevicePointer(&d, h, 0) == cudaSuccess) {
        if (ctx->h_stage) cudaFreeHost(ctx->h_stage);
        ctx->h_stage = (double *)h;
        ctx->h_stage_dev = (double *)d;
        ctx->stage_n = cap;
        return true;
    }
    cudaGetLastError();  // no page-locked memory to be had: by DMA
    if (h) cudaFreeHost(h);
    return false;
}

bool stream_capturing(dm_ctx *ctx) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(ctx->stream, &cs) != cudaSuccess) cudaGetLastError();
    return cs == cudaStreamCaptureStatusActive;
}

// First in every call that uses or changes the state.  What the host knows of
// the device (valid midpoint, boxes, filter bounds, order) holds neither for a call that is
// being captured, which runs when it is replayed, nor after one.  From the
// first such call on the position sets and the slot of the step counter stay
// where the recorded launches expect them (adopt_sets, leave_slot).
void cloud_enter(dm_cloud *c) {
    c->capturing = stream_capturing(c->ctx);
    if (c->capturing && !c->captured) {
        c->drop_graphs();
        c->captured = true;
    }
    if (!c->captured) return;
    c->state_changed(false);
    c->split_stale = true;
    c->order_dirty = true;
    c->dirty_upload = 0;
}

// Last in a call that steps: `slot` was current when it began.
template <class Owner>
int leave_slot(Owner *c, int slot) {
    if (c->captured && c->slot != slot) {
        DM_CUDA(c->ctx, launch_pdl(copy_slot, dim3(1), dim3(1), 0, c->ctx->stream, c->d, c->slot, slot));
        c->slot = slot;
    }
    return DM_OK;
}

}  // namespace

// ===========================================================================
// C ABI
// ===========================================================================
extern "C" {

int dm_version(void) { return DM_ABI_VERSION; }

int dm_ctx_create(int device, dm_ctx **out) {
    if (!out) {
        g_create_error = "dm_ctx_create: out is NULL";
        return DM_ERR_ARG;
    }
    *out = nullptr;
    int count = 0;
    cudaError_t e = cudaGetDeviceCount(&count);
    if (e != cudaSuccess || device < 0 || device >= count) {
        g_create_error = std::string("dm_ctx_create: no CUDA device ") + std::to_string(device) +
                         (e != cudaSuccess ? std::string(": ") + cudaGetErrorString(e) : std::string());
        return e != cudaSuccess ? DM_ERR_CUDA : DM_ERR_ARG;
    }
    dm_ctx *ctx = new dm_ctx();
    ctx->device = device;
    e = cudaSetDevice(device);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&ctx->own_stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&ctx->num_sms, cudaDevAttrMultiProcessorCount, device);
    int major = 0, minor = 0;
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, device);
    if (e != cudaSuccess) {
        g_create_error = std::string("dm_ctx_create: ") + cudaGetErrorString(e);
        delete ctx;
        return DM_ERR_CUDA;
    }
    if (major * 10 + minor != 103) {
        g_create_error = "dm_ctx_create: this build targets sm_103a (GB300); device is sm_" +
                         std::to_string(major) + std::to_string(minor);
        cudaStreamDestroy(ctx->own_stream);
        delete ctx;
        return DM_ERR_UNSUPPORTED;
    }
    ctx->stream = ctx->own_stream;
    *out = ctx;
    return DM_OK;
}

int dm_ctx_destroy(dm_ctx *ctx) {
    if (!ctx) return DM_ERR_ARG;
    cudaSetDevice(ctx->device);
    cudaStreamSynchronize(ctx->stream);
    for (auto &p : ctx->prof_events) {
        cudaEventDestroy(p.first);
        cudaEventDestroy(p.second);
    }
    if (ctx->own_stream) cudaStreamDestroy(ctx->own_stream);
    if (ctx->h_err) cudaFreeHost(ctx->h_err);
    if (ctx->h_adapt) cudaFreeHost(ctx->h_adapt);
    if (ctx->h_stage) cudaFreeHost(ctx->h_stage);
    if (ctx->stage_read) cudaEventDestroy(ctx->stage_read);
    delete ctx;
    return DM_OK;
}

int dm_ctx_set_stream(dm_ctx *ctx, void *stream) {
    if (!ctx) return DM_ERR_ARG;
    ctx->stream = (cudaStream_t)stream;  // NULL: the CUDA default (legacy) stream
    return DM_OK;
}

int dm_ctx_reset_stream(dm_ctx *ctx) {
    if (!ctx) return DM_ERR_ARG;
    ctx->stream = ctx->own_stream;
    return DM_OK;
}

int dm_ctx_synchronize(dm_ctx *ctx) {
    if (!ctx) return DM_ERR_ARG;
    DM_CUDA(ctx, cudaSetDevice(ctx->device));
    DM_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return DM_OK;
}

int dm_last_error(const dm_ctx *ctx, char *buf, size_t len) {
    if (!buf || len == 0) return DM_ERR_ARG;
    const std::string &s = ctx ? ctx->err : g_create_error;
    snprintf(buf, len, "%s", s.c_str());
    return DM_OK;
}

int dm_ctx_launch_count(dm_ctx *ctx, long long *count) {
    if (!ctx || !count) return DM_ERR_ARG;
    *count = ctx->launches;
    return DM_OK;
}

int dm_ctx_profile_enable(dm_ctx *ctx, int enable) {
    if (!ctx) return DM_ERR_ARG;
    ctx->prof = enable != 0;
    ctx->prof_used = 0;
    ctx->prof_pairs = 0.0;
    ctx->prof_launches = 0;
    return DM_OK;
}

int dm_ctx_profile_read(dm_ctx *ctx, double *total_ms, long long *launches, double *pairs) {
    if (!ctx) return DM_ERR_ARG;
    DM_CUDA(ctx, cudaSetDevice(ctx->device));
    DM_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    double tot = 0.0;
    for (size_t k = 0; k < ctx->prof_used; k++) {
        float ms = 0.0f;
        DM_CUDA(ctx, cudaEventElapsedTime(&ms, ctx->prof_events[k].first, ctx->prof_events[k].second));
        tot += ms;
    }
    if (total_ms) *total_ms = tot;
    if (launches) *launches = ctx->prof_launches;
    if (pairs) *pairs = ctx->prof_pairs;
    ctx->prof_used = 0;
    ctx->prof_pairs = 0.0;
    ctx->prof_launches = 0;
    return DM_OK;
}

int dm_probe_peak(dm_ctx *ctx, int kind, double *tflops) {
    if (!ctx || !tflops || (kind != 0 && kind != 1)) return DM_ERR_ARG;
    DM_CUDA(ctx, cudaSetDevice(ctx->device));
    void *out = nullptr;
    DM_CUDA(ctx, cudaMalloc(&out, 16));
    cudaEvent_t a, b;
    DM_CUDA(ctx, cudaEventCreate(&a));
    DM_CUDA(ctx, cudaEventCreate(&b));
    const int threads = 256, blocks = ctx->num_sms * 8;
    const int iters = (kind == 0) ? 8192 : 256;
    double best = 0.0;
    for (int rep = 0; rep < 4; rep++) {
        DM_CUDA(ctx, cudaEventRecord(a, ctx->stream));
        if (kind == 0)
            fma_probe<float><<<blocks, threads, 0, ctx->stream>>>((float *)out, iters, 0.999f, 0.001f);
        else
            fma_probe<double><<<blocks, threads, 0, ctx->stream>>>((double *)out, iters, 0.999, 0.001);
        DM_CUDA(ctx, cudaGetLastError());
        DM_CUDA(ctx, cudaEventRecord(b, ctx->stream));
        DM_CUDA(ctx, cudaEventSynchronize(b));
        float ms = 0.0f;
        DM_CUDA(ctx, cudaEventElapsedTime(&ms, a, b));
        const double flops = 2.0 * 16.0 * (double)iters * threads * (double)blocks;
        best = std::max(best, flops / (ms * 1e-3) / 1e12);
    }
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    cudaFree(out);
    *tflops = best;
    return DM_OK;
}

int dm_cloud_create(dm_ctx *ctx, int n, const double *x, const double *y, const double *vx,
                    const double *vy, const double *q, const double *m, dm_cloud **out) {
    if (!ctx || !out || n < 1 || !x || !y || !vx || !vy || !q || !m)
        return ctx ? ctx->fail(DM_ERR_ARG, "dm_cloud_create: bad argument") : DM_ERR_ARG;
    *out = nullptr;
    DM_CUDA(ctx, cudaSetDevice(ctx->device));
    dm_cloud *c = new dm_cloud();
    c->ctx = ctx;
    c->n = n;
    c->n_pad = (n + 63) & ~63;
    // a re-sort costs less than the pair sweeps it saves every step (a confined
    // cloud's particles cross many cutoffs per step while it collapses, close
    // pairs of a random cloud are thrown out, and a stale order inflates
    // every group box)
    c->reorder_interval = 1;
    c->coulomb = 1.0 / (4.0 * M_PI * 8.8541878E-12);
    c->d.coulomb = c->coulomb;
    c->d.rc2 = (10.0 / 2e4) * (10.0 / 2e4);  // default kappa until set_forces
    c->d.rc2_up = round_up_f32(c->d.rc2);
    const size_t nd = align256((size_t)c->n_pad * sizeof(double));
    const size_t nf4 = align256((size_t)c->n_pad * sizeof(float4));
    const size_t ni = align256((size_t)c->n_pad * sizeof(int));
    c->sort_blocks = (n + kSortPerBlock - 1) / kSortPerBlock;
    const size_t nh = align256((size_t)kSortBuckets * (c->sort_blocks + 1) * sizeof(uint32_t));
    const size_t ngb = align256((size_t)(c->n_pad / 32) * sizeof(float4));
    const size_t nsp = align256((size_t)(c->n_pad / 1024 + 1) * sizeof(float4));
    const size_t total = nd * (6 + 5 + 6 + 2 + 6) + nf4 * 8 + (ngb + nsp) * 4 + ni * 6 + nh + 1024 + 512 +
                         align256(sizeof(double) * 5 * (kDiagBlocks + 1)) +
                         align256(sizeof(float) * kMomentBlocks * kMomentFields);
    cudaError_t e = cudaMalloc(&c->block, total);
    if (e != cudaSuccess) {
        delete c;
        return ctx->fail(DM_ERR_NOMEM, "dm_cloud_create: cudaMalloc(%zu) failed: %s", total, cudaGetErrorString(e));
    }
    char *p = (char *)c->block;
    auto takeD = [&]() { double *r = (double *)p; p += nd; return r; };
    auto takeF4 = [&]() { float4 *r = (float4 *)p; p += nf4; return r; };
    c->d.n = n;
    c->d.n_pad = c->n_pad;
    c->d.x = takeD(); c->d.y = takeD(); c->d.vx = takeD(); c->d.vy = takeD();
    c->d.q = takeD(); c->d.m = takeD();
    for (int k = 0; k < 2; k++) { c->d.k1[k] = takeD(); c->d.k2[k] = takeD(); }
    c->d.invm = takeD();
    c->d.px[0] = c->d.x;  // position set 0 is the state
    c->d.py[0] = c->d.y;
    for (int b = 1; b < 4; b++) { c->d.px[b] = takeD(); c->d.py[b] = takeD(); }
    c->d_fx = takeD();
    c->d_fy = takeD();
    for (int b = 0; b < 4; b++) { c->d.pa[b] = takeF4(); c->d.pb[b] = takeF4(); }
    for (int b = 0; b < 4; b++) { c->d.gbox[b] = (float4 *)p; p += ngb; }
    for (int b = 0; b < 4; b++) {
        c->d.gsuper[b] = (c->n_pad / 32 >= kSuperMin) ? (float4 *)p : nullptr;
        p += nsp;
    }
    c->d.eval_pairs = (unsigned long long *)p; p += 256;
    c->d.step_ctr = (unsigned long long *)p; p += 256;
    c->d.time = (double *)(c->d.step_ctr + 4);  // same 256-byte slot, bytes 32-55
    c->d.err = (int *)p; p += 256;
    c->d_dt = (double *)p; p += 256;
    c->d_min = (unsigned int *)p; p += 256;
    auto takeI = [&]() { int *r = (int *)p; p += ni; return r; };
    c->d.orig = takeI();
    c->sort.keys[0] = (uint32_t *)takeI();
    c->sort.keys[1] = (uint32_t *)takeI();
    c->sort.vals[0] = takeI();
    c->sort.vals[1] = takeI();
    c->sort.orig_stage = takeI();
    for (int k = 0; k < 6; k++) c->sort.stage[k] = takeD();
    c->sort.hist = (uint32_t *)p; p += nh;
    c->sort.box = (double *)p; c->sort.keep = (int *)(p + 64);
    c->sort.changed = (int *)(p + 68);
    c->sort.order = (OrderRecord *)(p + 128); p += 256;

    c->sort.moments = (float *)p; p += align256(sizeof(float) * kMomentBlocks * kMomentFields);
    c->d_diag = (double *)p; p += align256(sizeof(double) * 5 * (kDiagBlocks + 1));
    cudaStream_t s = ctx->stream;
    const size_t bytes = (size_t)n * sizeof(double);
    e = cudaMemsetAsync(c->block, 0, total, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(c->d.x, x, bytes, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(c->d.y, y, bytes, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(c->d.vx, vx, bytes, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(c->d.vy, vy, bytes, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(c->d.q, q, bytes, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(c->d.m, m, bytes, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) {
        set_identity<<<(n + 255) / 256, 256, 0, s>>>(c->d.orig, n);
        init_positions<<<(c->n_pad + 255) / 256, 256, 0, s>>>(c->d);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        cudaFree(c->block);
        delete c;
        return ctx->fail(DM_ERR_CUDA, "dm_cloud_create: %s", cudaGetErrorString(e));
    }
    c->f.flags = kConfinement | kDrag | kShieldedCoulomb;
    c->f.shielding = 2e4;
    c->f.confine = 100;
    c->f.gamma = 10.0;
    *out = c;
    return DM_OK;
}

int dm_cloud_destroy(dm_cloud *c) {
    if (!c) return DM_ERR_ARG;
    cudaSetDevice(c->ctx->device);
    cudaStreamSynchronize(c->ctx->stream);
    c->drop_graphs();
    cudaFree(c->block);
    delete c;
    return DM_OK;
}

int dm_cloud_size(const dm_cloud *c, int *n) {
    if (!c || !n) return DM_ERR_ARG;
    *n = c->n;
    return DM_OK;
}

int dm_cloud_upload(dm_cloud *c, const double *x, const double *y, const double *vx, const double *vy) {
    if (!c) return DM_ERR_ARG;
    dm_ctx *ctx = c->ctx;
    if (!x || !y || !vx || !vy) return ctx->fail(DM_ERR_ARG, "dm_cloud_upload: NULL array");
    DM_CUDA(ctx, cudaSetDevice(ctx->device));
    cloud_enter(c);
    const size_t bytes = (size_t)c->n * sizeof(double);
    // caller order -> staging -> the cloud's current internal order (charges,
    // masses and the order stay; position set 0 and its boxes are rewritten)
    double **st = c->sort.stage;
    const StateBuffers B(x, y, vx, vy);
    if (B.viewed()) {
        copy4<<<(c->n + 255) / 256, 256, 0, ctx->stream>>>(c->n, B.view(0), B.view(1), B.view(2), B.view(3), st[0],
                                                           st[1], st[2], st[3], nullptr, nullptr);
        DM_CUDA(ctx, cudaGetLastError());
        ctx->launches += 1;
    } else if (staged_copies(ctx, c->n, B)) {
        const size_t n = (size_t)c->n;
        const double *in[4] = {x, y, vx, vy}, *d = ctx->h_stage_dev;
        DM_CUDA(ctx, cudaEventSynchronize(ctx->stage_read));
        for (int k = 0; k < 4; k++) std::memcpy(ctx->h_stage + k * n, in[k], bytes);
        copy4<<<(c->n + 255) / 256, 256, 0, ctx->stream>>>(c->n, d, d + n, d + 2 * n, d + 3 * n, st[0], st[1], st[2],
                                                           st[3], nullptr, nullptr);
        DM_CUDA(ctx, cudaGetLastError());
        DM_CUDA(ctx, cudaEventRecord(ctx->stage_read, ctx->stream));
        ctx->launches += 1;
    } else {
        DM_CUDA(ctx, cudaMemcpyAsync(st[0], x, bytes, cudaMemcpyHostToDevice, ctx->stream));
        DM_CUDA(ctx, cudaMemcpyAsync(st[1], y, bytes, cudaMemcpyHostToDevice, ctx->stream));
        DM_CUDA(ctx, cudaMemcpyAsync(st[2], vx, bytes, cudaMemcpyHostToDevice, ctx->stream));
        DM_CUDA(ctx, cudaMemcpyAsync(st[3], vy, bytes, cudaMemcpyHostToDevice, ctx->stream));
    }
    // the uploaded positions may be far from the old order
    if (!c->order_dirty) c->dirty_upload = ++c->uploads;
    c->order_dirty = true;
    upload_internal_order<<<(c->n_pad + 255) / 256, 256, 0, ctx->stream>>>(c->d, c->sort, c->dirty_upload);
    c->state_changed(true);
    DM_CUDA(ctx, cudaGetLastError());
    ctx->launches += 1;
    return DM_OK;
}

int dm_cloud_download(dm_cloud *c, double *x, double *y, double *vx, double *vy) {
    if (!c) return DM_ERR_ARG;
    dm_ctx *ctx = c->ctx;
    DM_CUDA(ctx, cudaSetDevice(ctx->device));
    const size_t bytes = (size_t)c->n * sizeof(double);
    double **st = c->sort.stage;
    scatter_to_caller<<<(c->n + 255) / 256, 256, 0, ctx->stream>>>(
        c->d.orig, c->n, c->d.x, c->d.y, c->d.vx, c->d.vy, st[0], st[1], st[2], st[3]);
    DM_CUDA(ctx, cudaGetLastError());
    ctx->launches++;
    // the error flags come back with the state: one synchronisation
    if (!ctx->h_err) DM_CUDA(ctx, cudaMallocHost((void **)&ctx->h_err, sizeof(int)));
    const StateBuffers B(x, y, vx, vy);
    int *err_dv = (int *)Buffer(ctx->h_err).view;
    if (B.viewed() && err_dv) {
        copy4<<<(c->n + 255) / 256, 256, 0, ctx->stream>>>(c->n, st[0], st[1], st[2], st[3], B.view(0), B.view(1),
                                                           B.view(2), B.view(3), c->d.err, err_dv);
        DM_CUDA(ctx, cudaGetLastError());
        ctx->launches++;
    } else if (err_dv && staged_copies(ctx, c->n, B)) {
        const size_t n = (size_t)c->n;
        const double *h = ctx->h_stage + 4 * (size_t)ctx->stage_n;
        double *d = ctx->h_stage_dev + 4 * (size_t)ctx->stage_n, *out[4] = {x, y, vx, vy};
        copy4<<<(c->n + 255) / 256, 256, 0, ctx->stream>>>(c->n, st[0], st[1], st[2], st[3], d, d + n, d + 2 * n,
                                                           d + 3 * n, c->d.err, err_dv);
        DM_CUDA(ctx, cudaGetLastError());
        ctx->launches++;
        DM_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        for (int k = 0; k < 4; k++)
            if (out[k]) std::memcpy(out[k], h + k * n, bytes);
        return device_error_status(ctx, c, *ctx->h_err);
    } else {
        if (x) DM_CUDA(ctx, cudaMemcpyAsync(x, st[0], bytes, cudaMemcpyDeviceToHost, ctx->stream));
        if (y) DM_CUDA(ctx, cudaMemcpyAsync(y, st[1], bytes, cudaMemcpyDeviceToHost, ctx->stream));
        if (vx) DM_CUDA(ctx, cudaMemcpyAsync(vx, st[2], bytes, cudaMemcpyDeviceToHost, ctx->stream));
        if (vy) DM_CUDA(ctx, cudaMemcpyAsync(vy, st[3], bytes, cudaMemcpyDeviceToHost, ctx->stream));
        DM_CUDA(ctx, cudaMemcpyAsync(ctx->h_err, c->d.err, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    }
    DM_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return device_error_status(ctx, c, *ctx->h_err);
}

int dm_cloud_set_charge_mass(dm_cloud *c, const double *q, const double *m) {
    if (!c) return DM_ERR_ARG;
    dm_ctx *ctx = c->ctx;
    DM_CUDA(ctx, cudaSetDevice(ctx->device));
    cloud_enter(c);
    const size_t bytes = (size_t)c->n * sizeof(double);
    double **st = c->sort.stage;
    // caller order -> staging -> internal order
    if (q) DM_CUDA(ctx, cudaMemcpyAsync(st[4], q, bytes, cudaMemcpyHostToDevice, ctx->stream));
    if (m) DM_CUDA(ctx, cudaMemcpyAsync(st[5], m, bytes, cudaMemcpyHostToDevice, ctx->stream));
    gather_from_caller<<<(c->n + 255) / 256, 256, 0, ctx->stream>>>(
        c->d.orig, c->n, q ? st[4] : nullptr, m ? st[5] : nullptr, c->d.q, c->d.m);
    // the float charge copy lives in the position sets: refresh set 0
    init_positions<<<(c->n_pad + 255) / 256, 256, 0, ctx->stream>>>(c->d);
    c->state_changed(false);
    DM_CUDA(ctx, cudaGetLastError());
    return DM_OK;
}

int dm_cloud_set_forces(dm_cloud *c, const dm_force_params *p) {
    if (!c || !p) return DM_ERR_ARG;
    dm_ctx *ctx = c->ctx;
    ForceParams fp;
    std::memcpy(&fp, p, sizeof(ForceParams));
    const char *why = nullptr;
    if (const int st = check_force_params(fp, &why))
        return ctx->fail(st, "dm_cloud_set_forces: %s (flags 0x%llx)", why, (unsigned long long)p->flags);
    cloud_enter(c);
    c->f = fp;
    c->d.rc2 = (p->shielding > 0.0) ? (10.0 / p->shielding) * (10.0 / p->shielding) : 0.0;
    c->d.rc2_up = round_up_f32(c->d.rc2);
    c->drop_graphs();
    // the position sets carry a per-particle filter bound that depends on kappa
    DM_CUDA(ctx, cudaSetDevice(ctx->device));
    init_positions<<<(c->n_pad + 255) / 256, 256, 0, ctx->stream>>>(c->d);
    c->state_changed(false);
    DM_CUDA(ctx, cudaGetLastError());
    return DM_OK;
}

int dm_cloud_eval_forces_device(dm_cloud *c, int precision, double *d_fx, double *d_fy) {
    if (!c) return DM_ERR_ARG;
    dm_ctx *ctx = c->ctx;
    if (precision != DM_FP64 && precision != DM_FP32C)
        return ctx->fail(DM_ERR_ARG, "bad precision %d", precision);
    DM_CUDA(ctx, cudaSetDevice(ctx->device));
    cloud_enter(c);
    if (c->order_dirty && wants_order(c->n, precision)) {  // spatial order first (internal only: outputs are in the caller's order)
        const int rc = reorder(c);
        if (rc) return rc;
    }
    int rc = ensure_tuned(c, precision);
    if (!rc) rc = launch_tuned(c, precision, make_stage_params(c, 0, kModeForceOnly, 0.0, nullptr));
    if (rc) return rc;
    const size_t bytes = (size_t)c->n * sizeof(double);
    if (d_fx && d_fx != c->d_fx) DM_CUDA(ctx, cudaMemcpyAsync(d_fx, c->d_fx, bytes, cudaMemcpyDeviceToDevice, ctx->stream));
    if (d_fy && d_fy != c->d_fy) DM_CUDA(ctx, cudaMemcpyAsync(d_fy, c->d_fy, bytes, cudaMemcpyDeviceToDevice, ctx->stream));
    return DM_OK;
}

int dm_cloud_eval_forces(dm_cloud *c, int precision, double *fx, double *fy) {
    if (!c) return DM_ERR_ARG;
    dm_ctx *ctx = c->ctx;
    if (!fx || !fy) return ctx->fail(DM_ERR_ARG, "dm_cloud_eval_forces: NULL output");
    int rc = dm_cloud_eval_forces_device(c, precision, nullptr, nullptr);
    if (rc) return rc;
    const size_t bytes = (size_t)c->n * sizeof(double);
    DM_CUDA(ctx, cudaMemcpyAsync(fx, c->d_fx, bytes, cudaMemcpyDeviceToHost, ctx->stream));
    DM_CUDA(ctx, cudaMemcpyAsync(fy, c->d_fy, bytes, cudaMemcpyDeviceToHost, ctx->stream));
    DM_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return DM_OK;
}

int dm_cloud_evaluated_pairs(dm_cloud *c, unsigned long long *pairs) {
    if (!c || !pairs) return c ? c->ctx->fail(DM_ERR_ARG, "dm_cloud_evaluated_pairs: NULL") : DM_ERR_ARG;
    dm_ctx *ctx = c->ctx;
    DM_CUDA(ctx, cudaSetDevice(ctx->device));
    DM_CUDA(ctx, cudaMemcpyAsync(pairs, c->d.eval_pairs, sizeof(unsigned long long), cudaMemcpyDeviceToHost,
                                 ctx->stream));
    DM_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return DM_OK;
}

int dm_cloud_eval_forces_stage(dm_cloud *c, int precision, int stage, double *fx, double *fy) {
    if (!c) return DM_ERR_ARG;
    if (stage < 1 || stage > 4) return c->ctx->fail(DM_ERR_ARG, "dm_cloud_eval_forces_stage: stage must be 1..4");
    c->eval_thermal_stage = stage;
    const int rc = dm_cloud_eval_forces(c, precision, fx, fy);
    c->eval_thermal_stage = 1;
    return rc;
}

int dm_cloud_step(dm_cloud *c, int nsteps, double dt, int precision, double *t_inout) {
    if (!c) return DM_ERR_ARG;
    dm_ctx *ctx = c->ctx;
    if (nsteps < 0 || !std::isfinite(dt)) return ctx->fail(DM_ERR_ARG, "dm_cloud_step: bad nsteps/dt");
    if (precision != DM_FP64 && precision != DM_FP32C)
        return ctx->fail(DM_ERR_ARG, "bad precision %d", precision);
    DM_CUDA(ctx, cudaSetDevice(ctx->device));
    cloud_enter(c);
    if (t_inout) {  // the force time of the first step is the caller's time
        set_time_slots<<<1, 1, 0, ctx->stream>>>(c->d.time, *t_inout);
        DM_CUDA(ctx, cudaGetLastError());
    }
    const int slot = c->slot;
    int rc = run_steps(c, nsteps, dt, precision);
    const int left = leave_slot(c, slot);
    if (rc || left) return rc ? rc : left;
    if (t_inout)
        for (int s = 0; s < nsteps; s++) *t_inout += dt;
    return DM_OK;
}

int dm_cloud_modify_timestep(dm_cloud *c, double init_dt, float *min_dist, double *dt_out) {
    if (!c) return DM_ERR_ARG;
    dm_ctx *ctx = c->ctx;
    if (c->n % 4 != 0 || c->n < 4)
        return ctx->fail(DM_ERR_ARG, "adaptive time step needs n %% 4 == 0 (Integrator.cpp:87-107)");
    DM_CUDA(ctx, cudaSetDevice(ctx->device));
    if (!ctx->h_adapt) DM_CUDA(ctx, cudaMallocHost((void **)&ctx->h_adapt, sizeof(AdaptiveResult)));
    AdaptiveResult *host = nullptr;
    DM_CUDA(ctx, cudaHostGetDevicePointer((void **)&host, ctx->h_adapt, 0));
    const int nb = c->n / 4, nt = (nb + kAdaptTile - 1) / kAdaptTile;
    const int blocks = (int)std::min<long long>((long long)nt * (nt + 1) / 2, (long long)ctx->num_sms * 8);
    float2 *pos = (float2 *)c->sort.stage[0];
    DM_CUDA(ctx, launch_pdl(adaptive_positions, dim3((c->n + 255) / 256), dim3(256), 0, ctx->stream, c->d, pos,
                            c->d_min));
    DM_CUDA(ctx, launch_pdl(checked_min_dist2, dim3(blocks), dim3(256), 0, ctx->stream, (const float2 *)pos, nb,
                            init_dt, c->d_min, c->d_dt, c->d.err, host));
    ctx->launches += 2;
    DM_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (min_dist) *min_dist = ctx->h_adapt->dmin;
    if (dt_out) *dt_out = ctx->h_adapt->dt;
    return device_error_status(ctx, c, ctx->h_adapt->err);
}

int dm_cloud_move_particles(dm_cloud *c, double end_time, double dt, int precision, int adaptive,
                            double *t_inout, int *steps) {
    if (!c || !t_inout) return c ? c->ctx->fail(DM_ERR_ARG, "t_inout is NULL") : DM_ERR_ARG;
    dm_ctx *ctx = c->ctx;
    if (!(dt > 0.0)) return ctx->fail(DM_ERR_ARG, "dt must be positive");
    double t = *t_inout;
    int count = 0;
    // the force time of the first step is the caller's time
    DM_CUDA(ctx, cudaSetDevice(ctx->device));
    cloud_enter(c);
    set_time_slots<<<1, 1, 0, ctx->stream>>>(c->d.time, t);
    DM_CUDA(ctx, cudaGetLastError());
    if (!adaptive) {
        // same accumulation as `while (currentTime < endTime) currentTime += dt`
        while (t < end_time) {
            t += dt;
            count++;
        }
        int rc = dm_cloud_step(c, count, dt, precision, nullptr);
        if (rc) return rc;
    } else {
        const int slot = c->slot;
        int rc = DM_OK;
        while (t < end_time) {
            double step_dt = 0.0;
            rc = reorder_if_due(c, precision, 0.0, false);
            if (!rc) rc = dm_cloud_modify_timestep(c, dt, nullptr, &step_dt);
            if (!rc) rc = launch_step(c, precision, 0.0, c->d_dt);
            if (rc) break;
            c->host_steps++;
            t += step_dt;
            count++;
        }
        const int left = leave_slot(c, slot);
        if (rc || left) return rc ? rc : left;
    }
    *t_inout = t;
    if (steps) *steps = count;
    return DM_OK;
}

int dm_cloud_diagnostics(dm_cloud *c, double out[5]) {
    if (!c || !out) return DM_ERR_ARG;
    dm_ctx *ctx = c->ctx;
    DM_CUDA(ctx, cudaSetDevice(ctx->device));
    const int blocks = diagnostics_blocks(c->n);
    const double kappa = c->f.shielding, rc = (kappa > 0.0) ? 10.0 / kappa : 0.0;
    diagnostics_partial<<<blocks, kDiagTile, 0, ctx->stream>>>(c->d, c->f, make_yukawa64(kappa, rc * rc), rc,
                                                               c->coulomb, c->d_diag);
    diagnostics_finish<<<1, 160, 0, ctx->stream>>>(c->d_diag, blocks, c->d_diag + 5 * kDiagBlocks);
    DM_CUDA(ctx, cudaGetLastError());
    ctx->launches += 2;
    DM_CUDA(ctx, cudaMemcpyAsync(out, c->d_diag + 5 * kDiagBlocks, 5 * sizeof(double), cudaMemcpyDeviceToHost,
                                 ctx->stream));
    DM_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return DM_OK;
}

int dm_ctx_set_autotune(dm_ctx *ctx, int enable) {
    if (!ctx) return DM_ERR_ARG;
    ctx->autotune = enable != 0;
    ctx->tune_cache.clear();
    return DM_OK;
}

int dm_cloud_autotune(dm_cloud *c, int precision, char *variant, size_t len, int *split) {
    if (!c) return DM_ERR_ARG;
    dm_ctx *ctx = c->ctx;
    if (precision != DM_FP64 && precision != DM_FP32C) return ctx->fail(DM_ERR_ARG, "bad precision %d", precision);
    DM_CUDA(ctx, cudaSetDevice(ctx->device));
    const int rc = ensure_tuned(c, precision);
    if (rc) return rc;
    const int pi = precision == DM_FP32C ? 1 : 0;
    if (variant && len) snprintf(variant, len, "%s", kVariants[c->tuned_variant[pi]].name);
    if (split) *split = c->split[pi];
    return DM_OK;
}

int dm_kernel_variants(char *buf, size_t len) {
    if (!buf || len == 0) return DM_ERR_ARG;
    std::string out;
    for (int v = 0; v < kNumVariants; v++) {
        if (v) out += ";";
        out += kVariants[v].name;
    }
    snprintf(buf, len, "%s", out.c_str());
    return DM_OK;
}

int dm_cloud_set_kernel(dm_cloud *c, const char *variant, int split) {
    if (!c || !variant) return DM_ERR_ARG;
    dm_ctx *ctx = c->ctx;
    if (std::strcmp(variant, "fp64<128,2,2,512>") == 0) variant = "fp64<4>";  // its name in earlier versions
    int vi = -1;
    for (int v = 0; v < kNumVariants; v++)
        if (std::strcmp(kVariants[v].name, variant) == 0) vi = v;
    if (vi < 0) return ctx->fail(DM_ERR_ARG, "unknown kernel variant '%s'", variant);
    const Variant &k = kVariants[vi];
    const int smax = k.cluster ? kMaxSplitCluster : kMaxSplitGlobal;
    if (split < 0 || split > smax) return ctx->fail(DM_ERR_ARG, "split %d outside [0, %d]", split, smax);
    DM_CUDA(ctx, cudaSetDevice(ctx->device));
    int rc = ensure_kernel_attrs(ctx);
    if (rc) return rc;
    if (split == 0) split = model_split(ctx, k, c->n, c->n_pad);
    if (k.cluster) {
        int nc = 0;
        cudaLaunchAttribute attr[2];
        cudaLaunchConfig_t cfg = make_cfg(ctx, k, (c->n + k.tile - 1) / k.tile, split, 2, attr);
        if (cudaOccupancyMaxActiveClusters(&nc, k.fn, &cfg) != cudaSuccess || nc <= 0) {
            cudaGetLastError();
            return ctx->fail(DM_ERR_UNSUPPORTED, "cluster of %d CTAs of %s cannot be scheduled", split, k.name);
        }
    } else {
        rc = ensure_partial(c, split);
        if (rc) return rc;
    }
    const int pi = k.precision == DM_FP32C ? 1 : 0;
    c->tuned_variant[pi] = vi;
    c->split[pi] = split;
    c->drop_graphs();
    return DM_OK;
}

int dm_cloud_set_reorder_interval(dm_cloud *c, int steps) {
    if (!c) return DM_ERR_ARG;
    if (steps < 0 || steps > kGraphSteps || (steps & (steps - 1)) != 0)
        return c->ctx->fail(DM_ERR_ARG, "reorder interval must be 0 or a power of two <= %d", kGraphSteps);
    c->reorder_interval = steps;
    c->keep_orders = false;
    c->drop_graphs();
    return DM_OK;
}

int dm_cloud_set_step_counter(dm_cloud *c, uint64_t step) {
    if (!c) return DM_ERR_ARG;
    dm_ctx *ctx = c->ctx;
    DM_CUDA(ctx, cudaSetDevice(ctx->device));
    unsigned long long v[2] = {step, step};
    DM_CUDA(ctx, cudaMemcpyAsync(c->d.step_ctr, v, sizeof(v), cudaMemcpyHostToDevice, ctx->stream));
    DM_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return DM_OK;
}

int dm_cloud_set_integrator(dm_cloud *c, int order) {
    if (!c) return DM_ERR_ARG;
    if (order != 2 && order != 4) return c->ctx->fail(DM_ERR_ARG, "integrator order must be 2 or 4");
    if (order != c->order) c->drop_graphs();
    c->order = order;
    return DM_OK;
}

int dm_cloud_set_time(dm_cloud *c, double t) {
    if (!c) return DM_ERR_ARG;
    dm_ctx *ctx = c->ctx;
    DM_CUDA(ctx, cudaSetDevice(ctx->device));
    set_time_slots<<<1, 1, 0, ctx->stream>>>(c->d.time, t);
    DM_CUDA(ctx, cudaGetLastError());
    return DM_OK;
}

int dm_cloud_get_time(dm_cloud *c, double *t) {
    if (!c || !t) return DM_ERR_ARG;
    dm_ctx *ctx = c->ctx;
    DM_CUDA(ctx, cudaSetDevice(ctx->device));
    double v = 0.0;
    DM_CUDA(ctx, cudaMemcpyAsync(&v, c->d.time + c->slot, sizeof(v), cudaMemcpyDeviceToHost, ctx->stream));
    DM_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    *t = v;
    return DM_OK;
}

int dm_cloud_get_step_counter(dm_cloud *c, uint64_t *step) {
    if (!c || !step) return DM_ERR_ARG;
    dm_ctx *ctx = c->ctx;
    DM_CUDA(ctx, cudaSetDevice(ctx->device));
    unsigned long long v = 0;
    DM_CUDA(ctx, cudaMemcpyAsync(&v, c->d.step_ctr + c->slot, sizeof(v), cudaMemcpyDeviceToHost, ctx->stream));
    DM_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    *step = v;
    return DM_OK;
}


// ===========================================================================
// Batched clouds
// ===========================================================================
}  // extern "C"

namespace {

struct BatchVariant {
    const char *name;
    bool cull;
    int nt, tile;
    size_t smem;
    const void *fn;
    cudaError_t (*launch)(const cudaLaunchConfig_t *, const StageParams &, const BatchCloud *, const BatchItem *);
};

template <int NW, int ILP, int TC, bool CULL>
cudaError_t launch_batch(const cudaLaunchConfig_t *cfg, const StageParams &P, const BatchCloud *desc,
                         const BatchItem *items) {
    return cudaLaunchKernelEx(cfg, batch_stage_fp32c<NW, ILP, TC, CULL>, P, desc, items);
}

#define DM_BATCH_VARIANT(NW, ILP, TC, CULL, SUFFIX)                                                \
    {"batch_fp32c<" #NW "," #ILP "," #TC SUFFIX ">", CULL, NW * 32, 32 * ILP,                      \
     Fp32cSmem<NW, ILP, TC>::bytes, (const void *)batch_stage_fp32c<NW, ILP, TC, CULL>,            \
     launch_batch<NW, ILP, TC, CULL>}

const BatchVariant kBatchVariants[] = {
    DM_BATCH_VARIANT(8, 4, 256, false, ""),
    DM_BATCH_VARIANT(4, 4, 256, false, ""),
    DM_BATCH_VARIANT(8, 2, 256, false, ""),
    DM_BATCH_VARIANT(4, 2, 128, false, ""),
    DM_BATCH_VARIANT(8, 4, 256, true, ",cull"),
    DM_BATCH_VARIANT(4, 2, 128, true, ",cull"),
    DM_BATCH_VARIANT(8, 2, 256, true, ",cull"),
};
constexpr int kNumBatchVariants = (int)(sizeof(kBatchVariants) / sizeof(kBatchVariants[0]));

}  // namespace

struct dm_batch {
    dm_ctx *ctx = nullptr;
    int nclouds = 0, total = 0, total_pad = 0;
    void *block = nullptr;
    CloudDev d{};
    std::vector<BatchCloud> hdesc;
    std::vector<int> hn;
    BatchCloud *ddesc = nullptr;
    int *dseg = nullptr;
    BatchItem *ditems[kNumBatchVariants] = {nullptr};
    int nitems[kNumBatchVariants] = {0};
    double *dbox = nullptr;  // [nclouds][8] key box and bounding box (batch_boxes)
    SortScratch sort{};
    int sort_blocks = 0;
    int mbits = 24;
    double *d_fx = nullptr, *d_fy = nullptr;
    float2 *partial = nullptr;  // [2 sets][2 axes][total_pad] pair sums of a pass
    int ngroups = 0;            // 32-particle groups over all clouds
    int *dgseg = nullptr;       // [ngroups] cloud of each group
    int variant = -1;
    int reorder_interval = 4;  // 1 when every cloud fits batch_sort_clouds
    int max_n = 0;             // largest cloud
    int order = 4;  // integrator: 4 = Runge_Kutta4, 2 = Runge_Kutta2
    bool order_dirty = true;
    bool boxes_valid[4] = {false, false, false, false};  // as dm_cloud's
    bool mid_valid = false;
    double mid_dt = 0.0;
    int slot = 0;
    bool capturing = false, captured = false;  // as dm_cloud's
    unsigned long long host_steps = 0;
    std::map<GraphKey, StepGraph> graphs;
    cudaStream_t graph_stream = nullptr;
    std::vector<void *> extra;

    void drop_graphs() {
        for (auto &kv : graphs) cudaGraphExecDestroy(kv.second.exec);
        graphs.clear();
    }
    ~dm_batch() {
        drop_graphs();
        for (void *p : extra) cudaFree(p);
        if (block) cudaFree(block);
    }
};

namespace {

// One pass of every cloud; mode kModeForceOnly: the forces at position set
// buf, evaluated nsets times.
int batch_launch_pass(dm_batch *B, int pass, int mode, double dt, int buf = 0, int nsets = 1) {
    dm_ctx *ctx = B->ctx;
    const BatchVariant &k = kBatchVariants[B->variant];
    StageParams P{};
    P.c = B->d;
    P.pass = pass;
    P.order = B->order;
    P.mode = mode;
    P.nsets = (mode == kModeForceOnly) ? nsets : 2;
    P.buf[0] = (mode == kModeForceOnly) ? buf : 2 * pass;
    P.buf[1] = (mode == kModeForceOnly) ? buf : 2 * pass + 1;
    P.slot = B->slot;
    P.therm_stage = 1;
    P.dt = dt;
    P.coulomb = B->d.coulomb;
    P.fx_out = B->d_fx;
    P.fy_out = B->d_fy;
    P.direct_min = direct_min_hits();
    P.near_direct_f2 = near_direct_f2();
    if (k.cull)
        for (int e = 0; e < P.nsets; e++) {
            const int b = P.buf[e];
            if (B->boxes_valid[b]) continue;
            DM_CUDA(ctx, launch_pdl(batch_group_bounds, dim3((B->ngroups * 32 + 255) / 256), dim3(256), 0, ctx->stream,
                                    B->d, (const BatchCloud *)B->ddesc, (const int *)B->dgseg, B->ngroups, b));
            ctx->launches++;
            B->boxes_valid[b] = true;
        }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(B->nitems[B->variant] * P.nsets);
    cfg.blockDim = dim3(k.nt);
    cfg.dynamicSmemBytes = k.smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    P.split = 1;
    P.partial = B->partial;
    DM_CUDA(ctx, k.launch(&cfg, P, B->ddesc, B->ditems[B->variant]));
    DM_CUDA(ctx, launch_pdl(batch_finish, dim3(B->ngroups), dim3(64), 0, ctx->stream, P, (const BatchCloud *)B->ddesc,
                            (const int *)B->dgseg));
    ctx->launches += 2;
    if (mode == kModeForceOnly) return DM_OK;
    const int ob = (pass == 0) ? 2 : 0;
    B->boxes_valid[ob] = B->boxes_valid[ob + 1] = true;
    if (P.order == 2) {
        if (B->captured) {
            DM_CUDA(ctx, launch_pdl(adopt_sets, dim3((B->total + 255) / 256), dim3(256), 0, ctx->stream, B->d,
                                    B->ngroups));
            ctx->launches++;
        } else {
            swap_sets(B->d);
        }
        B->boxes_valid[0] = B->boxes_valid[1] = true;
    }
    if (P.order == 2 || pass == 1) {
        B->mid_valid = true;
        B->mid_dt = dt;
        if (P.order == 2) B->slot ^= 1;
    }
    return DM_OK;
}

// Puts every cloud in Morton order; mid, force: as reorder's.
int batch_reorder(dm_batch *B, double dt = 0.0, bool mid = false, bool force = true) {
    dm_ctx *ctx = B->ctx;
    cudaStream_t s = ctx->stream;
    const int n = B->total;
    const int grid = (n + 255) / 256;
    SortScratch &z = B->sort;
    if (B->max_n <= kBatchSortMax) {  // one block per cloud sorts it in place
        DM_CUDA(ctx, cudaFuncSetAttribute(batch_sort_clouds, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)kBatchSortSmem));
        DM_CUDA(ctx, launch_pdl(batch_sort_clouds, dim3(B->nclouds), dim3(kBatchSortThreads), kBatchSortSmem, s,
                                B->d, (const BatchCloud *)B->ddesc, B->dbox, dt, mid,
                                B->mid_valid && B->mid_dt == dt && B->boxes_valid[1], force || !B->boxes_valid[0], B->slot,
                                B->sort.order));
        ctx->launches++;
        B->boxes_valid[0] = true;
        B->boxes_valid[1] = B->mid_valid = mid;
        B->mid_dt = dt;
        B->order_dirty = false;
        return DM_OK;
    }
    batch_boxes<<<B->nclouds, 256, 0, s>>>(B->d.x, B->d.y, B->ddesc, B->dbox);
    batch_keys<<<grid, 256, 0, s>>>(B->d.x, B->d.y, n, B->dseg, B->dbox, B->mbits, z.keys[0], z.vals[0]);
    const int bits = B->mbits + 32 - __builtin_clz((unsigned)std::max(B->nclouds - 1, 1));
    DM_CUDA(ctx, cudaGetLastError());
    int cur = 0;
    int rc = radix_passes(ctx, z, n, B->sort_blocks, bits, false, nullptr, &cur);
    if (rc) return rc;
    DM_CUDA(ctx, launch_pdl(permute_gather, dim3(grid), dim3(256), 0, s, B->d, (const int *)z.vals[cur], z,
                            (const int *)nullptr));
    DM_CUDA(ctx, launch_pdl(batch_commit, dim3((B->total_pad + 255) / 256), dim3(256), 0, s, B->d,
                            (const BatchCloud *)B->ddesc, (const int *)B->dseg, z));
    ctx->launches += 4;
    B->boxes_valid[0] = B->boxes_valid[1] = B->mid_valid = false;
    B->order_dirty = false;
    return DM_OK;
}

int batch_enqueue_steps(dm_batch *B, int nsteps, double dt) {
    dm_ctx *ctx = B->ctx;
    for (int s = 0; s < nsteps; s++) {
        if (B->order_dirty || (B->reorder_interval > 0 && B->host_steps % (unsigned)B->reorder_interval == 0)) {
            int rc = batch_reorder(B, dt, true, B->order_dirty || B->reorder_interval != 1);
            if (rc) return rc;
        }
        if (!B->mid_valid || B->mid_dt != dt) {
            DM_CUDA(ctx, launch_pdl(batch_midpoint, dim3((B->total + 255) / 256), dim3(256), 0, ctx->stream, B->d,
                                    (const BatchCloud *)B->ddesc, (const int *)B->dseg, dt));
            ctx->launches++;
            B->boxes_valid[1] = false;
            B->mid_valid = true;
            B->mid_dt = dt;
        }
        for (int pass = 0; pass < B->order / 2; pass++) {
            int rc = batch_launch_pass(B, pass, kModeStep, dt);
            if (rc) return rc;
        }
        B->host_steps++;
    }
    return DM_OK;
}

int batch_tune(dm_batch *B) {
    dm_ctx *ctx = B->ctx;
    int rc = DM_OK;
    for (int v = 0; v < kNumBatchVariants; v++) {
        const BatchVariant &k = kBatchVariants[v];
        DM_CUDA(ctx, cudaFuncSetAttribute(k.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)k.smem));
        // work items (cloud, tile), largest clouds first
        std::vector<BatchItem> items;
        std::vector<int> order(B->nclouds);
        for (int c = 0; c < B->nclouds; c++) order[c] = c;
        std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return B->hn[a] > B->hn[b]; });
        for (int c : order)
            for (int t = 0; t * k.tile < B->hn[c]; t++) items.push_back({c, t, B->hdesc[c].off, B->hn[c]});
        B->nitems[v] = (int)items.size();
        if (!B->ditems[v]) {
            DM_CUDA(ctx, cudaMalloc((void **)&B->ditems[v], items.size() * sizeof(BatchItem)));
            B->extra.push_back(B->ditems[v]);
        }
        DM_CUDA(ctx, cudaMemcpyAsync(B->ditems[v], items.data(), items.size() * sizeof(BatchItem),
                                     cudaMemcpyHostToDevice, ctx->stream));
    }
    int best = 0;
    if (ctx->autotune) {
        if (B->order_dirty) {  // tune on the particle order the steps will see
            rc = batch_reorder(B);
            if (rc) return rc;
        }
        // two states, as for one cloud: the batch as it is (buffer 0) and
        // every cloud squeezed to ~30% in-cutoff pairs (buffer 1)
        batch_tune_compress<<<(B->total + 255) / 256, 256, 0, ctx->stream>>>(B->d, B->ddesc, B->dseg, B->dbox);
        B->boxes_valid[1] = B->mid_valid = false;
        DM_CUDA(ctx, cudaGetLastError());
        cudaEvent_t a, b;
        DM_CUDA(ctx, cudaEventCreate(&a));
        DM_CUDA(ctx, cudaEventCreate(&b));
        float best_ms = 1e30f;
        std::vector<int> candidates;  // culling variants first (see tune_precision)
        for (const bool cull : {true, false})
            for (int v = 0; v < kNumBatchVariants; v++)
                if (kBatchVariants[v].cull == cull) candidates.push_back(v);
        for (const int v : candidates) {
            B->variant = v;
            float total = 0.0f, ms_state[2] = {0.0f, 0.0f};
            for (int st = 0; st < 2 && total < 1.3f * best_ms; st++) {
                float one = 1e30f;
                for (int r = 0; r < 3; r++) {  // best of three
                    if (total + kTuneWeight[st] * std::min(one, 1e6f) * (r > 0) >= 1.3f * best_ms) break;
                    DM_CUDA(ctx, cudaEventRecord(a, ctx->stream));
                    rc = batch_launch_pass(B, 0, kModeForceOnly, 0.0, st, 2);
                    if (rc) return rc;
                    DM_CUDA(ctx, cudaEventRecord(b, ctx->stream));
                    DM_CUDA(ctx, cudaEventSynchronize(b));
                    float ms = 0.0f;
                    DM_CUDA(ctx, cudaEventElapsedTime(&ms, a, b));
                    one = std::min(one, ms);
                }
                total += kTuneWeight[st] * one;
                ms_state[st] = one;
            }
            if (tune_verbose())
                fprintf(stderr, "dm autotune batch %s: %.4f ms (state) %.4f ms (dense copy)\n", kBatchVariants[v].name,
                        ms_state[0], ms_state[1]);
            if (total < best_ms) {
                best_ms = total;
                best = v;
            }
        }
        cudaEventDestroy(a);
        cudaEventDestroy(b);
    }
    B->variant = best;
    return DM_OK;
}

// First in every call that uses the state: as cloud_enter.
void batch_enter(dm_batch *B) {
    B->capturing = stream_capturing(B->ctx);
    if (B->capturing && !B->captured) {
        B->drop_graphs();
        B->captured = true;
    }
    if (!B->captured) return;
    B->boxes_valid[0] = B->boxes_valid[1] = B->mid_valid = false;
    B->order_dirty = true;
}

// nsteps of every cloud, in captured blocks where there are enough (see run_steps).
int batch_run_steps(dm_batch *B, int nsteps, double dt) {
    dm_ctx *ctx = B->ctx;
    if (ctx->prof || B->capturing || nsteps < kGraphSteps) return batch_enqueue_steps(B, nsteps, dt);
    if (B->graph_stream != ctx->stream) {
        B->drop_graphs();
        B->graph_stream = ctx->stream;
    }
    while (nsteps > 0 && (B->order_dirty || (B->reorder_interval > 0 && B->host_steps % kGraphSteps != 0))) {
        int rc = batch_enqueue_steps(B, 1, dt);
        if (rc) return rc;
        nsteps--;
    }
    if (nsteps < kGraphSteps) return batch_enqueue_steps(B, nsteps, dt);
    const bool sorts = B->reorder_interval > 0 && B->max_n <= kBatchSortMax;
    // what the captured steps start from: see run_steps
    if (sorts ? !B->boxes_valid[0] : !(B->mid_valid && B->mid_dt == dt)) {
        int rc = batch_enqueue_steps(B, 1, dt);
        return rc ? rc : batch_run_steps(B, nsteps - 1, dt);
    }
    const GraphKey key{DM_FP32C, kGraphSteps, dt, B->slot};
    auto it = B->graphs.find(key);
    if (it == B->graphs.end()) {
        cudaGraph_t g = nullptr;
        const unsigned long long saved = B->host_steps;
        const long long sl = ctx->launches;
        if (sorts) B->mid_valid = false;
        const CloudDev state = B->d;
        const int slot = B->slot;
        DM_CUDA(ctx, cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
        int rc = batch_enqueue_steps(B, kGraphSteps, dt);
        cudaError_t ec = cudaStreamEndCapture(ctx->stream, &g);
        B->host_steps = saved;
        const long long launches = ctx->launches - sl;
        ctx->launches = sl;
        if (rc || ec != cudaSuccess) {  // see run_steps
            B->d = state;
            B->slot = slot;
            B->boxes_valid[0] = B->boxes_valid[1] = B->mid_valid = false;
        }
        if (rc) {
            if (g) cudaGraphDestroy(g);
            return rc;
        }
        if (ec != cudaSuccess) return ctx->fail(DM_ERR_CUDA, "graph capture failed: %s", cudaGetErrorString(ec));
        cudaGraphExec_t ge = nullptr;
        ec = cudaGraphInstantiate(&ge, g, 0);
        cudaGraphDestroy(g);
        if (ec != cudaSuccess) return ctx->fail(DM_ERR_CUDA, "graph instantiate failed: %s", cudaGetErrorString(ec));
        it = B->graphs.emplace(key, StepGraph{ge, launches}).first;
    }
    const int reps = nsteps / kGraphSteps;
    for (int r = 0; r < reps; r++) {
        DM_CUDA(ctx, cudaGraphLaunch(it->second.exec, ctx->stream));
        B->host_steps += kGraphSteps;
        ctx->launches += it->second.launches;
        B->mid_valid = true;
        B->mid_dt = dt;
        for (bool &v : B->boxes_valid) v = true;
    }
    return batch_enqueue_steps(B, nsteps - reps * kGraphSteps, dt);
}

}  // namespace

extern "C" {

int dm_batch_create(dm_ctx *ctx, int nclouds, const int *n, const double *x, const double *y,
                    const double *vx, const double *vy, const double *q, const double *m,
                    const dm_force_params *params, dm_batch **out) {
    if (!ctx || !out || nclouds < 1 || !n || !x || !y || !vx || !vy || !q || !m || !params)
        return ctx ? ctx->fail(DM_ERR_ARG, "dm_batch_create: bad argument") : DM_ERR_ARG;
    if (nclouds > 65536) return ctx->fail(DM_ERR_ARG, "dm_batch_create: at most 65536 clouds");
    *out = nullptr;
    long long total = 0;
    for (int c = 0; c < nclouds; c++) {
        if (n[c] < 1) return ctx->fail(DM_ERR_ARG, "dm_batch_create: cloud %d has n = %d", c, n[c]);
        ForceParams fp;
        std::memcpy(&fp, &params[c], sizeof(ForceParams));
        const char *why = nullptr;
        if (const int st = check_force_params(fp, &why))
            return ctx->fail(st, "dm_batch_create: cloud %d: %s", c, why);
        total += n[c];
    }
    if (total > (1LL << 30)) return ctx->fail(DM_ERR_ARG, "dm_batch_create: too many particles");
    DM_CUDA(ctx, cudaSetDevice(ctx->device));
    dm_batch *B = new dm_batch();
    B->ctx = ctx;
    B->nclouds = nclouds;
    B->total = (int)total;
    B->total_pad = ((int)total + 63) & ~63;
    B->hn.assign(n, n + nclouds);
    B->max_n = *std::max_element(n, n + nclouds);
    // per-cloud sort in one launch: cheap enough to keep every cloud's order
    // fresh each step (confined clouds collapse and their groups spread)
    B->reorder_interval = (B->max_n <= kBatchSortMax) ? 1 : 4;
    const int cbits = 32 - __builtin_clz((unsigned)std::max(nclouds - 1, 1));
    B->mbits = std::min(24, (32 - cbits) & ~1);
    const double coulomb = 1.0 / (4.0 * M_PI * 8.8541878E-12);
    const int np = B->total_pad;
    const size_t nd = align256((size_t)np * sizeof(double));
    const size_t nf4 = align256((size_t)np * sizeof(float4));
    const size_t ni = align256((size_t)np * sizeof(int));
    B->sort_blocks = (B->total + kSortPerBlock - 1) / kSortPerBlock;
    const size_t nh = align256((size_t)kSortBuckets * (B->sort_blocks + 1) * sizeof(uint32_t));
    const size_t ndesc = align256((size_t)nclouds * sizeof(BatchCloud));
    const size_t nbb = align256((size_t)nclouds * 8 * sizeof(double));
    const size_t nord = align256((size_t)nclouds * sizeof(OrderRecord));
    const size_t bytes_total = nd * (6 + 5 + 6 + 2 + 6) + nf4 * 8 + ni * 7 + nh + ndesc + nbb + nord + 1024;
    cudaError_t e = cudaMalloc(&B->block, bytes_total);
    if (e != cudaSuccess) {
        delete B;
        return ctx->fail(DM_ERR_NOMEM, "dm_batch_create: cudaMalloc(%zu): %s", bytes_total, cudaGetErrorString(e));
    }
    char *p = (char *)B->block;
    auto takeD = [&]() { double *r = (double *)p; p += nd; return r; };
    auto takeF4 = [&]() { float4 *r = (float4 *)p; p += nf4; return r; };
    auto takeI = [&]() { int *r = (int *)p; p += ni; return r; };
    CloudDev &d = B->d;
    d.n = B->total;
    d.n_pad = np;
    d.coulomb = coulomb;
    d.x = takeD(); d.y = takeD(); d.vx = takeD(); d.vy = takeD(); d.q = takeD(); d.m = takeD();
    for (int k = 0; k < 2; k++) { d.k1[k] = takeD(); d.k2[k] = takeD(); }
    d.invm = takeD();
    d.px[0] = d.x;  // position set 0 is the state
    d.py[0] = d.y;
    for (int b = 1; b < 4; b++) { d.px[b] = takeD(); d.py[b] = takeD(); }
    B->d_fx = takeD();
    B->d_fy = takeD();
    for (int k = 0; k < 6; k++) B->sort.stage[k] = takeD();
    for (int b = 0; b < 4; b++) { d.pa[b] = takeF4(); d.pb[b] = takeF4(); }
    d.orig = takeI();
    B->dseg = takeI();
    B->sort.keys[0] = (uint32_t *)takeI();
    B->sort.keys[1] = (uint32_t *)takeI();
    B->sort.vals[0] = takeI();
    B->sort.vals[1] = takeI();
    B->sort.orig_stage = takeI();
    B->sort.hist = (uint32_t *)p; p += nh;
    B->ddesc = (BatchCloud *)p; p += ndesc;
    B->dbox = (double *)p; p += nbb;
    B->sort.order = (OrderRecord *)p; p += nord;
    d.step_ctr = (unsigned long long *)p; p += 256;
    d.time = (double *)(d.step_ctr + 4);  // same 256-byte slot, bytes 32-55
    d.err = (int *)p; p += 256;
    // host descriptors
    B->hdesc.resize(nclouds);
    std::vector<int> seg((size_t)B->total), orig((size_t)B->total), gseg;
    int off = 0;
    for (int c = 0; c < nclouds; c++) {
        BatchCloud &bc = B->hdesc[c];
        bc.off = off;
        bc.n = n[c];
        bc.goff = B->ngroups;
        for (int g = 0; g < (n[c] + 31) / 32; g++) gseg.push_back(c);
        B->ngroups += (n[c] + 31) / 32;
        std::memcpy(&bc.f, &params[c], sizeof(ForceParams));
        const double kappa = params[c].shielding;
        bc.rc2 = (kappa > 0.0) ? (10.0 / kappa) * (10.0 / kappa) : 0.0;
        bc.rc2_up = round_up_f32(bc.rc2);
        bc.rc2_lo = (float)(bc.rc2 * (1.0 - 4e-6));
        bc.rc2_hi = (float)(bc.rc2 * (1.0 + 4e-6));
        bc.kappa_f = (float)kappa;
        bc.nkl2e = (float)(-kappa * 1.4426950408889634);
        for (int i = 0; i < n[c]; i++) {
            seg[off + i] = c;
            orig[off + i] = off + i;
        }
        off += n[c];
    }
    cudaStream_t s = ctx->stream;
    // group boxes (culling kernels), the group -> cloud map, the swept-pair counter
    for (int b = 0; b < 4 && e == cudaSuccess; b++) {
        e = cudaMalloc((void **)&d.gbox[b], (size_t)B->ngroups * sizeof(float4));
        if (e == cudaSuccess) B->extra.push_back(d.gbox[b]);
    }
    if (e == cudaSuccess) e = cudaMalloc((void **)&B->partial, (size_t)4 * np * sizeof(float2));
    if (e == cudaSuccess) B->extra.push_back(B->partial);
    if (e == cudaSuccess) e = cudaMalloc((void **)&B->dgseg, gseg.size() * sizeof(int));
    if (e == cudaSuccess) B->extra.push_back(B->dgseg);
    if (e == cudaSuccess) e = cudaMalloc((void **)&d.eval_pairs, sizeof(unsigned long long));
    if (e == cudaSuccess) B->extra.push_back(d.eval_pairs);
    if (e == cudaSuccess) e = cudaMemsetAsync(d.eval_pairs, 0, sizeof(unsigned long long), s);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(B->dgseg, gseg.data(), gseg.size() * sizeof(int), cudaMemcpyHostToDevice, s);
    const size_t bt = (size_t)B->total * sizeof(double);
    if (e == cudaSuccess) e = cudaMemsetAsync(B->block, 0, bytes_total, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d.x, x, bt, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d.y, y, bt, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d.vx, vx, bt, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d.vy, vy, bt, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d.q, q, bt, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d.m, m, bt, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(B->dseg, seg.data(), seg.size() * sizeof(int), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d.orig, orig.data(), orig.size() * sizeof(int), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(B->ddesc, B->hdesc.data(), nclouds * sizeof(BatchCloud), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) {
        batch_init_positions<<<(np + 255) / 256, 256, 0, s>>>(d, B->ddesc, B->dseg);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        delete B;
        return ctx->fail(DM_ERR_CUDA, "dm_batch_create: %s", cudaGetErrorString(e));
    }
    int rc = batch_tune(B);
    if (rc) {
        delete B;
        return rc;
    }
    *out = B;
    return DM_OK;
}

int dm_batch_destroy(dm_batch *B) {
    if (!B) return DM_ERR_ARG;
    cudaSetDevice(B->ctx->device);
    cudaStreamSynchronize(B->ctx->stream);
    delete B;
    return DM_OK;
}

int dm_batch_step(dm_batch *B, int nsteps, double dt, int precision) {
    if (!B) return DM_ERR_ARG;
    dm_ctx *ctx = B->ctx;
    if (precision != DM_FP32C)
        return ctx->fail(DM_ERR_UNSUPPORTED, "batched clouds run the FP32C kernel; step FP64 clouds singly");
    if (nsteps < 0 || !std::isfinite(dt)) return ctx->fail(DM_ERR_ARG, "dm_batch_step: bad nsteps/dt");
    DM_CUDA(ctx, cudaSetDevice(ctx->device));
    batch_enter(B);
    const int slot = B->slot;
    const int rc = batch_run_steps(B, nsteps, dt), left = leave_slot(B, slot);
    return rc ? rc : left;
}

int dm_batch_eval_forces(dm_batch *B, int precision, double *fx, double *fy) {
    if (!B || !fx || !fy) return B ? B->ctx->fail(DM_ERR_ARG, "NULL output") : DM_ERR_ARG;
    dm_ctx *ctx = B->ctx;
    if (precision != DM_FP32C)
        return ctx->fail(DM_ERR_UNSUPPORTED, "batched clouds run the FP32C kernel");
    DM_CUDA(ctx, cudaSetDevice(ctx->device));
    batch_enter(B);
    int rc = batch_launch_pass(B, 0, kModeForceOnly, 0.0);
    if (rc) return rc;
    const size_t bt = (size_t)B->total * sizeof(double);
    DM_CUDA(ctx, cudaMemcpyAsync(fx, B->d_fx, bt, cudaMemcpyDeviceToHost, ctx->stream));
    DM_CUDA(ctx, cudaMemcpyAsync(fy, B->d_fy, bt, cudaMemcpyDeviceToHost, ctx->stream));
    DM_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return DM_OK;
}

int dm_batch_download(dm_batch *B, double *x, double *y, double *vx, double *vy) {
    if (!B) return DM_ERR_ARG;
    dm_ctx *ctx = B->ctx;
    DM_CUDA(ctx, cudaSetDevice(ctx->device));
    const size_t bt = (size_t)B->total * sizeof(double);
    double **st = B->sort.stage;
    scatter_to_caller<<<(B->total + 255) / 256, 256, 0, ctx->stream>>>(
        B->d.orig, B->total, B->d.x, B->d.y, B->d.vx, B->d.vy, st[0], st[1], st[2], st[3]);
    DM_CUDA(ctx, cudaGetLastError());
    ctx->launches++;
    if (x) DM_CUDA(ctx, cudaMemcpyAsync(x, st[0], bt, cudaMemcpyDeviceToHost, ctx->stream));
    if (y) DM_CUDA(ctx, cudaMemcpyAsync(y, st[1], bt, cudaMemcpyDeviceToHost, ctx->stream));
    if (vx) DM_CUDA(ctx, cudaMemcpyAsync(vx, st[2], bt, cudaMemcpyDeviceToHost, ctx->stream));
    if (vy) DM_CUDA(ctx, cudaMemcpyAsync(vy, st[3], bt, cudaMemcpyDeviceToHost, ctx->stream));
    DM_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    int h = 0;
    DM_CUDA(ctx, cudaMemcpy(&h, B->d.err, sizeof(int), cudaMemcpyDeviceToHost));
    if (h) {
        cudaMemset(B->d.err, 0, sizeof(int));
        return ctx->fail(DM_ERR_NUMERIC, "non-finite particle position in the batch");
    }
    return DM_OK;
}

int dm_batch_variants(char *buf, size_t len) {
    if (!buf || len == 0) return DM_ERR_ARG;
    std::string out;
    for (int v = 0; v < kNumBatchVariants; v++) {
        if (v) out += ";";
        out += kBatchVariants[v].name;
    }
    snprintf(buf, len, "%s", out.c_str());
    return out.size() < len ? DM_OK : DM_ERR_ARG;
}

int dm_batch_set_kernel(dm_batch *B, const char *variant) {
    if (!B || !variant) return B ? B->ctx->fail(DM_ERR_ARG, "dm_batch_set_kernel: NULL") : DM_ERR_ARG;
    for (int v = 0; v < kNumBatchVariants; v++)
        if (std::strcmp(kBatchVariants[v].name, variant) == 0) {
            B->variant = v;
            B->drop_graphs();
            return DM_OK;
        }
    return B->ctx->fail(DM_ERR_ARG, "dm_batch_set_kernel: unknown variant '%s'", variant);
}

int dm_batch_evaluated_pairs(dm_batch *B, unsigned long long *pairs) {
    if (!B || !pairs) return B ? B->ctx->fail(DM_ERR_ARG, "dm_batch_evaluated_pairs: NULL") : DM_ERR_ARG;
    dm_ctx *ctx = B->ctx;
    DM_CUDA(ctx, cudaSetDevice(ctx->device));
    DM_CUDA(ctx, cudaMemcpyAsync(pairs, B->d.eval_pairs, sizeof(unsigned long long), cudaMemcpyDeviceToHost,
                                 ctx->stream));
    DM_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return DM_OK;
}

int dm_batch_info(dm_batch *B, char *variant, size_t len, int *nitems, int *grid) {
    if (!B) return DM_ERR_ARG;
    if (variant && len) snprintf(variant, len, "%s", kBatchVariants[B->variant].name);
    if (nitems) *nitems = B->nitems[B->variant];
    if (grid) *grid = 2 * B->nitems[B->variant];  // a block per position set
    return DM_OK;
}

int dm_batch_set_integrator(dm_batch *B, int order) {
    if (!B) return DM_ERR_ARG;
    if (order != 2 && order != 4) return B->ctx->fail(DM_ERR_ARG, "integrator order must be 2 or 4");
    if (order != B->order) B->drop_graphs();
    B->order = order;
    return DM_OK;
}

int dm_batch_set_time(dm_batch *B, double t) {
    if (!B) return DM_ERR_ARG;
    dm_ctx *ctx = B->ctx;
    DM_CUDA(ctx, cudaSetDevice(ctx->device));
    set_time_slots<<<1, 1, 0, ctx->stream>>>(B->d.time, t);
    DM_CUDA(ctx, cudaGetLastError());
    return DM_OK;
}

int dm_batch_get_time(dm_batch *B, double *t) {
    if (!B || !t) return DM_ERR_ARG;
    dm_ctx *ctx = B->ctx;
    DM_CUDA(ctx, cudaSetDevice(ctx->device));
    double v = 0.0;
    DM_CUDA(ctx, cudaMemcpyAsync(&v, B->d.time + B->slot, sizeof(v), cudaMemcpyDeviceToHost, ctx->stream));
    DM_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    *t = v;
    return DM_OK;
}

int dm_batch_set_step_counter(dm_batch *B, uint64_t step) {
    if (!B) return DM_ERR_ARG;
    dm_ctx *ctx = B->ctx;
    unsigned long long v[2] = {step, step};
    DM_CUDA(ctx, cudaMemcpy(B->d.step_ctr, v, sizeof(v), cudaMemcpyHostToDevice));
    return DM_OK;
}


// ===========================================================================
// Differentiable rollout support: FP64 forces and their VJP on device arrays
// ===========================================================================
}  // extern "C"

struct dm_adjoint {
    dm_ctx *ctx = nullptr;
    int nclouds = 0, total = 0, nblocks = 0;
    std::vector<AdjCloud> hdesc;
    AdjCloud *ddesc = nullptr;
    int *dcloud = nullptr, *dtile = nullptr;
    double coulomb = 0.0;
    // fused RK4 step and adjoint: one block of total-length arrays
    void *work = nullptr;
    double *k1[4], *k23[4], *pbuf[2][4], *dk[2][4], *mu[3][4], *ax[2], *ay[2], *invm;
    AdjSplit split[2];
    // FP64 kernels: 32-particle groups (cloud, tile), largest clouds first, in
    // clusters of `csize` blocks
    int ngroups = 0, csize = 1;
    int2 *dgroups = nullptr;
    ~dm_adjoint() {
        if (dgroups) cudaFree(dgroups);
        if (ddesc) cudaFree(ddesc);
        if (dcloud) cudaFree(dcloud);
        if (dtile) cudaFree(dtile);
        if (work) cudaFree(work);
    }
};

namespace {
void adj_fill(dm_adjoint *A, const dm_force_params *params) {
    for (int c = 0; c < A->nclouds; c++) {
        AdjCloud &d = A->hdesc[c];
        d.flags = params[c].flags;
        d.kappa = params[c].shielding;
        d.confine = params[c].confine;
        d.confine_x = params[c].confine_x;
        d.confine_y = params[c].confine_y;
        d.gamma = params[c].gamma;
        d.rc2 = (d.kappa > 0.0) ? (10.0 / d.kappa) * (10.0 / d.kappa) : 0.0;
        d.rc2_up = round_up_f32(d.rc2);
        d.rc2_lo = (float)(d.rc2 * (1.0 - 4e-6));
        d.rc2_hi = (float)(d.rc2 * (1.0 + 4e-6));
        d.kappa_f = (float)d.kappa;
        d.kappa2_f = (float)(d.kappa * d.kappa);
        kappa_log2e(d.kappa, d.kl2e_hi, d.kl2e_lo);
        d.nkl2e = (float)(-d.kappa * 1.4426950408889634);
        d.y64 = make_yukawa64(d.kappa, d.rc2);
    }
}

// Launch of an FP64 group kernel over every 32-particle group.
template <int NS, typename... KArgs, typename... Args>
cudaError_t adj_launch64(dm_adjoint *A, void (*kernel)(KArgs...), Args &&...args) {
    constexpr int smem = (int)sizeof(AdjGroupSmem<NS>);
    cudaError_t e = cudaFuncSetAttribute((const void *)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(A->ngroups * A->csize);
    cfg.blockDim = dim3(32 * kAdjWarps);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = A->ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = A->csize;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

cudaError_t adj_launch_prepare(dm_adjoint *A, const AdjPrepareIO &R) {
    adj_prepare<<<A->nblocks, kAdjThreads, 0, A->ctx->stream>>>(A->ddesc, A->dcloud, A->dtile, R);
    A->ctx->launches++;
    return cudaGetLastError();
}

// Forces (MODE 0) or their VJP (MODE 1) alone.
template <int MODE>
cudaError_t adj_launch_once(dm_adjoint *A, int precision, const AdjOnce &O) {
    A->ctx->launches++;
    if (precision == DM_FP32C) {
        adjoint_kernel<MODE><<<A->nblocks, kAdjThreads, 0, A->ctx->stream>>>(A->ddesc, A->dcloud, A->dtile, O,
                                                                             A->coulomb);
        return cudaGetLastError();
    }
    // no scratch: such calls may be queued on several streams at once
    return adj_launch64<(MODE == 0 ? 2 : 4)>(A, adj_once_fp64<MODE>, (const AdjCloud *)A->ddesc,
                                             (const int2 *)A->dgroups, O, A->coulomb);
}
}  // namespace

extern "C" {

int dm_adjoint_create(dm_ctx *ctx, int nclouds, const int *n, const dm_force_params *params,
                      dm_adjoint **out) {
    if (!ctx || !out || nclouds < 1 || !n || !params) return ctx ? ctx->fail(DM_ERR_ARG, "dm_adjoint_create: bad argument") : DM_ERR_ARG;
    const long long known = kConfinement | kDrag | kShieldedCoulomb | kRectConfinement;
    for (int c = 0; c < nclouds; c++) {
        if (n[c] < 1) return ctx->fail(DM_ERR_ARG, "dm_adjoint_create: cloud %d is empty", c);
        if (params[c].flags & ~known)
            return ctx->fail(DM_ERR_UNSUPPORTED, "dm_adjoint_create: only confinement, drag and shielded "
                                                 "Coulomb forces are differentiated");
        ForceParams fp;
        std::memcpy(&fp, &params[c], sizeof(ForceParams));
        const char *why = nullptr;
        if (const int st = check_force_params(fp, &why))
            return ctx->fail(st, "dm_adjoint_create: cloud %d: %s", c, why);
    }
    DM_CUDA(ctx, cudaSetDevice(ctx->device));
    dm_adjoint *A = new dm_adjoint();
    A->ctx = ctx;
    A->nclouds = nclouds;
    A->coulomb = 1.0 / (4.0 * M_PI * 8.8541878E-12);
    A->hdesc.resize(nclouds);
    std::vector<int> bc, bt;
    int off = 0;
    for (int c = 0; c < nclouds; c++) {
        A->hdesc[c].off = off;
        A->hdesc[c].n = n[c];
        for (int t = 0; t * kAdjThreads < n[c]; t++) {
            bc.push_back(c);
            bt.push_back(t);
        }
        off += n[c];
    }
    A->total = off;
    A->nblocks = (int)bc.size();
    adj_fill(A, params);
    std::vector<int> order(nclouds);
    for (int c = 0; c < nclouds; c++) order[c] = c;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return n[a] > n[b]; });
    std::vector<int2> groups;
    for (int c : order)
        for (int t = 0; 32 * t < n[c]; t++) groups.push_back(make_int2(c, t));
    A->ngroups = (int)groups.size();
    // enough blocks for four on every SM, each warp at least one j group of
    // the largest cloud
    A->csize = std::min({8, (4 * ctx->num_sms + A->ngroups - 1) / A->ngroups,
                         std::max(1, (n[order[0]] + 32 * kAdjWarps - 1) / (32 * kAdjWarps))});
    cudaError_t e = cudaMalloc((void **)&A->ddesc, nclouds * sizeof(AdjCloud));
    if (e == cudaSuccess) e = cudaMalloc((void **)&A->dcloud, bc.size() * sizeof(int));
    if (e == cudaSuccess) e = cudaMalloc((void **)&A->dtile, bt.size() * sizeof(int));
    if (e == cudaSuccess) e = cudaMemcpy(A->ddesc, A->hdesc.data(), nclouds * sizeof(AdjCloud), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(A->dcloud, bc.data(), bc.size() * sizeof(int), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(A->dtile, bt.data(), bt.size() * sizeof(int), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMalloc((void **)&A->dgroups, groups.size() * sizeof(int2));
    if (e == cudaSuccess)
        e = cudaMemcpy(A->dgroups, groups.data(), groups.size() * sizeof(int2), cudaMemcpyHostToDevice);
    // scratch of the fused RK4 step and its adjoint: 41 arrays of total
    // doubles, 2 of float4 and 4 of float2
    const size_t nd = align256((size_t)A->total * sizeof(double));
    const size_t nf4 = align256((size_t)A->total * sizeof(float4));
    if (e == cudaSuccess) e = cudaMalloc(&A->work, (41 + 4) * nd + 2 * nf4);
    if (e == cudaSuccess) {
        char *p = (char *)A->work;
        auto take = [&]() { double *r = (double *)p; p += nd; return r; };
        for (int c = 0; c < 4; c++) A->k1[c] = take();
        for (int c = 0; c < 4; c++) A->k23[c] = take();
        for (int b = 0; b < 2; b++)
            for (int c = 0; c < 4; c++) A->pbuf[b][c] = take();
        for (int b = 0; b < 2; b++)
            for (int c = 0; c < 4; c++) A->dk[b][c] = take();
        for (int b = 0; b < 3; b++)
            for (int c = 0; c < 4; c++) A->mu[b][c] = take();
        for (int b = 0; b < 2; b++) {
            A->ax[b] = take();
            A->ay[b] = take();
            A->split[b].l = (float2 *)take();
            A->split[b].a = (float2 *)take();
        }
        A->invm = take();
        for (int b = 0; b < 2; b++) {
            A->split[b].p = (float4 *)p;
            p += nf4;
        }
    }
    if (e != cudaSuccess) {
        delete A;
        return ctx->fail(DM_ERR_CUDA, "dm_adjoint_create: %s", cudaGetErrorString(e));
    }
    *out = A;
    return DM_OK;
}

int dm_adjoint_destroy(dm_adjoint *A) {
    if (!A) return DM_ERR_ARG;
    cudaSetDevice(A->ctx->device);
    cudaStreamSynchronize(A->ctx->stream);
    delete A;
    return DM_OK;
}

int dm_adjoint_set_params(dm_adjoint *A, const dm_force_params *params) {
    if (!A || !params) return DM_ERR_ARG;
    dm_ctx *ctx = A->ctx;
    adj_fill(A, params);
    DM_CUDA(ctx, cudaSetDevice(ctx->device));
    DM_CUDA(ctx, cudaMemcpyAsync(A->ddesc, A->hdesc.data(), A->nclouds * sizeof(AdjCloud),
                                 cudaMemcpyHostToDevice, ctx->stream));
    DM_CUDA(ctx, cudaStreamSynchronize(ctx->stream));  // the host copy may be reused at once
    return DM_OK;
}

int dm_adjoint_forces(dm_adjoint *A, int precision, const double *x, const double *y, const double *vx,
                      const double *vy, const double *q, const double *m, double *fx, double *fy,
                      double *fpx, double *fpy) {
    if (!A || !x || !y || !vx || !vy || !q || !m || !fx || !fy) return A ? A->ctx->fail(DM_ERR_ARG, "NULL pointer") : DM_ERR_ARG;
    dm_ctx *ctx = A->ctx;
    if (precision != DM_FP64 && precision != DM_FP32C)
        return ctx->fail(DM_ERR_ARG, "dm_adjoint_forces: unknown precision %d", precision);
    DM_CUDA(ctx, cudaSetDevice(ctx->device));
    DM_CUDA(ctx, adj_launch_once<0>(A, precision, AdjOnce{x, y, vx, vy, q, m, nullptr, nullptr, {fx, fy, fpx, fpy}}));
    return DM_OK;
}

int dm_adjoint_rk4_step(dm_adjoint *A, int precision, double dt, double *x, double *y, double *vx, double *vy,
                        const double *q, const double *m, double *stages) {
    if (!A || !x || !y || !vx || !vy || !q || !m) return A ? A->ctx->fail(DM_ERR_ARG, "NULL pointer") : DM_ERR_ARG;
    dm_ctx *ctx = A->ctx;
    if (precision != DM_FP64 && precision != DM_FP32C)
        return ctx->fail(DM_ERR_ARG, "dm_adjoint_rk4_step: unknown precision %d", precision);
    if (!std::isfinite(dt)) return ctx->fail(DM_ERR_ARG, "dm_adjoint_rk4_step: dt must be finite");
    DM_CUDA(ctx, cudaSetDevice(ctx->device));
    const size_t n = (size_t)A->total;
    double *base[4] = {x, y, vx, vy};
    if (stages)
        for (int c = 0; c < 4; c++)
            DM_CUDA(ctx, cudaMemcpyAsync(stages + c * n, base[c], n * sizeof(double), cudaMemcpyDeviceToDevice,
                                         ctx->stream));
    AdjPrepareIO R{};
    R.x = x;
    R.y = y;
    R.m = m;
    R.out = A->split[0];
    R.invm = A->invm;
    DM_CUDA(ctx, adj_launch_prepare(A, R));
    for (int st = 1; st <= 4; st++) {
        AdjStepIO io{};
        double *in[4];
        for (int c = 0; c < 4; c++) {
            in[c] = (st == 1) ? base[c] : stages ? stages + (4 * (st - 1) + c) * n : A->pbuf[st & 1][c];
            io.next[c] = (st == 4) ? nullptr : stages ? stages + (4 * st + c) * n : A->pbuf[(st + 1) & 1][c];
            io.s[c] = base[c];
            io.k1[c] = A->k1[c];
            io.k23[c] = A->k23[c];
        }
        io.x = in[0]; io.y = in[1]; io.vx = in[2]; io.vy = in[3];
        io.in = A->split[(st - 1) & 1];
        io.out = A->split[st & 1];
        io.q = q;
        io.m = m;
        io.invm = A->invm;
        io.dt = dt;
        io.stage = st;
        if (precision == DM_FP32C) {
            adj_step_fp32c<<<A->nblocks, kAdjThreads, 0, ctx->stream>>>(A->ddesc, A->dcloud, A->dtile, io, A->coulomb);
            DM_CUDA(ctx, cudaGetLastError());
        } else {
            DM_CUDA(ctx, adj_launch64<2>(A, adj_step_fp64, (const AdjCloud *)A->ddesc, (const int2 *)A->dgroups, io,
                                         A->coulomb));
        }
        ctx->launches++;
    }
    return DM_OK;
}

int dm_adjoint_rk4_step_vjp(dm_adjoint *A, int precision, double dt, const double *stages, const double *q,
                            const double *m, double *lx, double *ly, double *lvx, double *lvy, double *gq,
                            double *gkappa, double *gkc) {
    if (!A || !stages || !q || !m || !lx || !ly || !lvx || !lvy || !gq || !gkappa || !gkc)
        return A ? A->ctx->fail(DM_ERR_ARG, "NULL pointer") : DM_ERR_ARG;
    dm_ctx *ctx = A->ctx;
    if (precision != DM_FP64 && precision != DM_FP32C)
        return ctx->fail(DM_ERR_ARG, "dm_adjoint_rk4_step_vjp: unknown precision %d", precision);
    if (!std::isfinite(dt)) return ctx->fail(DM_ERR_ARG, "dm_adjoint_rk4_step_vjp: dt must be finite");
    DM_CUDA(ctx, cudaSetDevice(ctx->device));
    const size_t n = (size_t)A->total;
    double *lam[4] = {lx, ly, lvx, lvy};
    AdjPrepareIO R{};
    R.x = stages + 12 * n;
    R.y = stages + 13 * n;
    R.m = m;
    R.out = A->split[0];
    R.invm = A->invm;
    R.ax = A->ax[0];
    R.ay = A->ay[0];
    R.dt = dt;
    for (int c = 0; c < 4; c++) {
        R.lam[c] = lam[c];
        R.dk[c] = A->dk[1][c];
    }
    DM_CUDA(ctx, adj_launch_prepare(A, R));
    for (int st = 4; st >= 1; st--) {
        AdjVjpIO V{};
        V.x = stages + (4 * (st - 1) + 0) * n;
        V.y = stages + (4 * (st - 1) + 1) * n;
        if (st > 1) {
            V.xn = stages + (4 * (st - 2) + 0) * n;
            V.yn = stages + (4 * (st - 2) + 1) * n;
        }
        const int rd = (st == 3 || st == 1) ? 1 : 0, wr = rd ^ 1;  // split positions and force adjoints
        V.in = A->split[rd];
        V.out = A->split[wr];
        V.ax = A->ax[rd];
        V.ay = A->ay[rd];
        V.axn = A->ax[wr];
        V.ayn = A->ay[wr];
        // dk_4 in dk[1], dk_3 in dk[0], dk_2 in dk[1], dk_1 in dk[0]
        for (int c = 0; c < 4; c++) {
            V.dk[c] = A->dk[rd ^ 1][c];
            V.dkn[c] = A->dk[wr ^ 1][c];
            V.lam[c] = lam[c];
            for (int b = 0; b < 3; b++) V.mu[b][c] = A->mu[b][c];
        }
        V.gq = gq;
        V.gkappa = gkappa;
        V.gkc = gkc;
        V.q = q;
        V.m = m;
        V.invm = A->invm;
        V.dt = dt;
        V.stage = st;
        if (precision == DM_FP32C) {
            adj_vjp_fp32c<<<A->nblocks, kAdjThreads, 0, ctx->stream>>>(A->ddesc, A->dcloud, A->dtile, V, A->coulomb);
            DM_CUDA(ctx, cudaGetLastError());
        } else {
            DM_CUDA(ctx, adj_launch64<4>(A, adj_vjp_fp64, (const AdjCloud *)A->ddesc, (const int2 *)A->dgroups, V,
                                         A->coulomb));
        }
        ctx->launches++;
    }
    return DM_OK;
}

int dm_adjoint_vjp(dm_adjoint *A, int precision, const double *x, const double *y, const double *vx,
                   const double *vy, const double *q, const double *m, const double *ax, const double *ay,
                   double *gx, double *gy, double *gvx, double *gvy, double *gq, double *gkappa, double *gkc) {
    if (!A || !x || !y || !vx || !vy || !q || !m || !ax || !ay || !gx || !gy || !gvx || !gvy || !gq ||
        !gkappa || !gkc)
        return A ? A->ctx->fail(DM_ERR_ARG, "NULL pointer") : DM_ERR_ARG;
    dm_ctx *ctx = A->ctx;
    if (precision != DM_FP64 && precision != DM_FP32C)
        return ctx->fail(DM_ERR_ARG, "dm_adjoint_vjp: unknown precision %d", precision);
    DM_CUDA(ctx, cudaSetDevice(ctx->device));
    DM_CUDA(ctx, adj_launch_once<1>(A, precision,
                                    AdjOnce{x, y, vx, vy, q, m, ax, ay, {gx, gy, gvx, gvy, gq, gkappa, gkc}}));
    return DM_OK;
}

}  // extern "C"
