// gx_dop853.cuh -- what the DOP853 orbit kernels share (gx_dop853.cu,
// gx_dop853_axis.cu): their arguments, the controller's scalars and the cluster
// operations of the batch-wide sums.
#pragma once

#include "gx_host.h"

namespace gx {

struct DopArgs {
    double atol, rtol, dt_max;
    int64_t nmax, nstiff;
    int64_t ntimes, out_stride, n_out;
    int32_t save_all, nbatch;
    const int32_t *cancel;  // host cancel flag (mapped memory) or nullptr
};

__device__ __forceinline__ double sign_d(double a, double b) { return (b < 0.0) ? -fabs(a) : fabs(a); }
__device__ __forceinline__ double min_d(double a, double b) { return (a < b) ? a : b; }
__device__ __forceinline__ double max_d(double a, double b) { return (a > b) ? a : b; }

// The larger magnitude, by integer comparison (a double comparison is an FP64-pipe instruction).
__device__ __forceinline__ double max_abs(double a, double b) {
    const long long m = 0x7fffffffffffffffLL, x = __double_as_longlong(a) & m, y = __double_as_longlong(b) & m;
    return __longlong_as_double(x > y ? x : y);
}

// The counters after a NaN step size: no later step is accepted, so gala evaluates
// eleven stages and rejects, up to nmax + 1 steps, and returns -2 (the state and the
// stored rows stay as they are).  A batch ends at once with what that comes to; the
// steps themselves are 1e6 by default, about a minute that no cancellation reaches.
__device__ __forceinline__ void nan_steps(int64_t nmax, int64_t naccpt, int64_t &nstep, int64_t &nfcn, int64_t &nrejct) {
    const int64_t left = nmax + 1 - nstep;
    nstep += left;
    nfcn += 11 * left;
    if (naccpt >= 1) nrejct += left;
}

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
// 8 bytes into the shared memory of CTA `rank` of the cluster, at this CTA's address p
__device__ __forceinline__ void cluster_store(double *p, unsigned rank, double v) {
    unsigned a, r;
    a = (unsigned)__cvta_generic_to_shared(p);
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(r), "d"(v) : "memory");
}

// DOP853 with one coordinate per lane (gx_dop853_axis.cu): whether the call is one
// for it, and its launch.
bool dop853_axis_takes(const DevPot &dp, const DevFrame &df, const DopArgs &A, int64_t n);
int launch_dop853_axis(const DevPot &dp, const DevFrame &df, const DopArgs &A, const double *w0, int64_t n, const double *t,
                       double *out, int32_t *status, int64_t *stats, cudaStream_t st);

}  // namespace gx
