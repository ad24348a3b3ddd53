// dm_noalloc.cu -- diagnostics entry point that allocates no memory.
//
// Some callers can't call cudaMalloc: a host application that manages every
// byte of device memory through its own fixed pool or budget, or code that
// must not trigger cudaMalloc's implicit device-wide synchronisation while
// its other streams run.  They already hold the particle state in their own
// device buffers and want the FP64 energies and momentum of it without
// creating a dm_cloud (which allocates ~350 bytes per particle).
//
// This file gives them dm_diagnostics_noalloc: the same diagnostics kernel,
// with its per-block partial sums in a fixed-size file-scope device array.
// Every GPU that loads this library holds that array (kDiagBlocks * 5
// doubles = 24 KiB) until the process exits.  Calls share the array, so
// calls that overlap on the GPU (different streams, or different host
// threads on the same device) race on it and must be serialised by the
// caller.  Each call overwrites every partial it later reads, so nothing has
// to start at zero.
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>

#include "../../include/demon_gb300.h"
#include "dm_misc.cuh"

using namespace dm;

namespace {

constexpr int kMaxParticles = 524288;  // the interface's limit (the scratch holds the blocks of any size)

// The scratch: one row of 5 partial sums per block (diagnostics_blocks: at most kDiagBlocks).
static __device__ __align__(256) double g_diag_scratch[kDiagBlocks * 5];

// In host code g_diag_scratch names a host-side stand-in, not device memory:
// the device address is looked up on every call, with the calling device
// current (see scratch_for_current_device).

// The device address of the scratch on the current device.  Looked up on
// every call rather than cached: the lookup allocates nothing, and a cached
// address would dangle after the host application calls cudaDeviceReset
// (the module is loaded again and the array may move).  The first call on a
// device may load this library's module there, so make that first call
// before any stream capture.
int scratch_for_current_device(double **out) {
    void *p = nullptr;
    if (cudaGetSymbolAddress(&p, g_diag_scratch) != cudaSuccess || !p) return DM_ERR_CUDA;
    *out = static_cast<double *>(p);
    return DM_OK;
}

}  // namespace

extern "C" int dm_diagnostics_noalloc(int n, const double *d_x, const double *d_y,
                                      const double *d_vx, const double *d_vy,
                                      const double *d_q, const double *d_m,
                                      const dm_force_params *params, double *d_out,
                                      void *stream) {
    // Errors are reported by status code only (no message store is shared
    // with the rest of the library, and building one would allocate).
    if (n < 1 || n > kMaxParticles) return DM_ERR_ARG;  // the scratch holds kMaxBlocks blocks
    if (!d_x || !d_y || !d_vx || !d_vy || !d_q || !d_m || !d_out || !params) return DM_ERR_ARG;
    ForceParams f;
    static_assert(sizeof(ForceParams) == sizeof(dm_force_params), "layout");
    memcpy(&f, params, sizeof(f));
    const char *why = nullptr;
    if (const int st = check_force_params(f, &why)) return st;  // same rules as dm_cloud_set_forces
    double *scratch = nullptr;
    const int rc = scratch_for_current_device(&scratch);
    if (rc) return rc;

    CloudDev c{};
    c.n = n;
    c.n_pad = n;
    c.x = const_cast<double *>(d_x);
    c.y = const_cast<double *>(d_y);
    c.vx = const_cast<double *>(d_vx);
    c.vy = const_cast<double *>(d_vy);
    c.q = const_cast<double *>(d_q);
    c.m = const_cast<double *>(d_m);
    const double coulomb = 1.0 / (4.0 * M_PI * 8.8541878E-12);
    const double cutoff = (f.shielding > 0.0) ? 10.0 / f.shielding : 0.0;
    const int blocks = diagnostics_blocks(n);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    diagnostics_partial<<<blocks, kDiagTile, 0, s>>>(c, f, make_yukawa64(f.shielding, cutoff * cutoff), cutoff, coulomb,
                                                     scratch);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) {
        diagnostics_finish<<<1, 160, 0, s>>>(scratch, blocks, d_out);
        e = cudaGetLastError();
    }
    return e == cudaSuccess ? DM_OK : DM_ERR_CUDA;
}
