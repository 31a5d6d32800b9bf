// gx_fixed.cu -- FP64 Leapfrog and Ruth4, one thread per orbit.
//
// Each thread carries its orbit's state in registers for the whole run and
// evaluates the composite gradient in registers (no per-step kernel launch, no
// state round trip through memory).  Snapshots go straight to gala's
// (6, ntimes, N) layout: at every step a warp writes 6 fully coalesced 256-byte
// rows.  The per-orbit arithmetic is gala's, expression by expression:
//   leapfrog  c_init_velocity / c_leapfrog_step (leapfrog.pyx:24-51,99-116)
//   ruth4     c_ruth4_step with gala's coefficients (ruth4.pyx:24-35,65-78,98-108)
// What bounds them is the FP64 pipe: one warp alone on a scheduler retires an
// FP64 instruction per 64 cycles whatever it depends on, and the SM's unit one per
// 19.  Roots and quotients run on the integer pipe (gx_device.cuh), Ruth4's
// zero-weight gradient is left out where it is certainly finite, Leapfrog's
// synchronised velocity is formed only where it is stored, and few orbits take four
// lanes each: 16,384 uneven orbits (100 to 2,000 steps) 69.8 -> 11.9 ms, 1,024
// Hernquist orbits x 1,000 stored steps 2.37 -> 0.73 ms, with the same bits (ln, in
// NFW, within an ulp).
#include "gx_host.h"
#include "gx_queue.cuh"
#include "gx_scf.cuh"

namespace gx {

struct Ruth4Coef {
    double c[4], d[4];
};

template <bool SCF>
__device__ __forceinline__ void grad_impl(const DevPot &pot, const double *x, double *g) {
    V3 q;
    q.v[0] = x[0]; q.v[1] = x[1]; q.v[2] = x[2];
    const V3 r = gradient_call<SCF>(pot, q);
    g[0] = r.v[0]; g[1] = r.v[1]; g[2] = r.v[2];
}
#define grad(pot, x, g) grad_impl<SCF>(pot, x, g)

// gala's v - g * dt / 2 from gd = g * dt: halving is exact, so the fused form
// rounds once, as the subtraction does.
__device__ __forceinline__ double half_kick(double v, double gd) { return fma(-0.5, gd, v); }

// One Ruth4 step (c_ruth4_step).  The first sub-step has d = 0, yet gala still
// evaluates the gradient there: a non-finite gradient (an orbit sitting on a
// singular point) turns v into NaN through 0 * inf.  Where the gradient is finite
// for certain (finite_gradient, and a step of ordinary size) the product is zero
// and the evaluation is left out: a quarter of the step.
template <bool SCF>
__device__ __forceinline__ void ruth4_step(const DevPot &pot, const Ruth4Coef &co, double dt, bool dt_ok, double *w) {
    double g[3];
    for (int s = 0; s < 4; s++) {
        if (s > 0 || !(dt_ok && finite_gradient(pot, w))) {
            grad(pot, w, g);
            for (int k = 0; k < 3; k++) w[3 + k] = w[3 + k] - co.d[s] * g[k] * dt;
        }
        for (int k = 0; k < 3; k++) w[k] = w[k] + co.c[s] * w[3 + k] * dt;
    }
}

template <bool SAVE_ALL, bool SCF>
__global__ void __launch_bounds__(128, 1) leapfrog_kernel(const __grid_constant__ DevPot pot, const double *__restrict__ w0, int64_t n,
                                                       const double *__restrict__ t, int64_t ntimes,
                                                       double *__restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double x[3], v[3], vh[3], g[3];
    for (int k = 0; k < 3; k++) {
        x[k] = w0[k * n + i];
        v[k] = w0[(3 + k) * n + i];
    }
    const double dt = t[1] - t[0];
    if (SAVE_ALL) {
        for (int k = 0; k < 3; k++) {
            out[(k * ntimes) * n + i] = x[k];
            out[((3 + k) * ntimes) * n + i] = v[k];
        }
    }
    // c_init_velocity: v_{1/2} = v - grad * dt / 2
    grad(pot, x, g);
    for (int k = 0; k < 3; k++) vh[k] = half_kick(v[k], g[k] * dt);
    for (int64_t j = 1; j < ntimes; j++) {
        // c_leapfrog_step: drift, gradient, half kick (output v), full kick
        for (int k = 0; k < 3; k++) x[k] = x[k] + vh[k] * dt;
        grad(pot, x, g);
        for (int k = 0; k < 3; k++) {
            const double gd = g[k] * dt;
            // v is an output only: formed where it is stored
            if (SAVE_ALL || j == ntimes - 1) v[k] = half_kick(vh[k], gd);
            vh[k] = vh[k] - gd;
        }
        if (SAVE_ALL) {
            for (int k = 0; k < 3; k++) {
                __stcs(&out[(k * ntimes + j) * n + i], x[k]);
                __stcs(&out[((3 + k) * ntimes + j) * n + i], v[k]);
            }
        }
    }
    if (!SAVE_ALL) {
        for (int k = 0; k < 3; k++) {
            out[k * n + i] = x[k];
            out[(3 + k) * n + i] = v[k];
        }
    }
}

template <bool SAVE_ALL, bool SCF>
__global__ void __launch_bounds__(128, 1) ruth4_kernel(const __grid_constant__ DevPot pot, Ruth4Coef co, const double *__restrict__ w0,
                                                    int64_t n, const double *__restrict__ t, int64_t ntimes,
                                                    double *__restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double w[6];
    for (int k = 0; k < 6; k++) w[k] = w0[k * n + i];
    const double dt = t[1] - t[0];
    const bool dt_ok = ordinary(dt);
    if (SAVE_ALL)
        for (int k = 0; k < 6; k++) out[(k * ntimes) * n + i] = w[k];
    for (int64_t j = 1; j < ntimes; j++) {
        ruth4_step<SCF>(pot, co, dt, dt_ok, w);
        if (SAVE_ALL)
            for (int k = 0; k < 6; k++) __stcs(&out[(k * ntimes + j) * n + i], w[k]);
    }
    if (!SAVE_ALL)
        for (int k = 0; k < 6; k++) out[k * n + i] = w[k];
}

// ---------------------------------------------------------------------------
// The same two integrators for few orbits: four lanes per orbit, one coordinate
// each (the fourth repeats z).  An FP64 instruction costs a warp 64 cycles whether
// one lane or 32 take part, and few orbits leave most of the schedulers without a
// warp, so the three coordinates of an orbit go side by side: per Leapfrog step of a
// Hernquist orbit 15 FP64 instructions instead of 36, of the MW composite 36 instead
// of 66.  The operations and their order are those above, so the bits are too.
// The line lies at one warp per scheduler (8 orbits per warp, 4 schedulers per SM):
// a Ruth4 step of 4,864 MW orbits takes 5.0 us, of 6,000 with one lane per orbit 10.9;
// 1,024 Hernquist orbits x 1,000 stored Leapfrog steps 1.80 -> 0.73 ms.
// ---------------------------------------------------------------------------
// gradient_axis's MODE for a potential.
static int axis_mode(const DevPot &dp) { return dp.sphere == GX_POT_HERNQUIST ? 1 : dp.dbh_order ? 1 + dp.dbh_order : 0; }

// Steps of the orbits of a warp's eight groups of four lanes, (x, v) the lane's
// coordinate: n_steps for each (EVEN, the same for all) or the lane's own ns <= n_steps,
// after which it goes along without moving.  store(j) after step j when SAVE.  The
// straight run serves from the first step on; where it declines a point, the warp is
// finished with the general form.
template <int MODE, bool RUTH, bool EVEN, bool SAVE, typename Store>
__device__ __forceinline__ void axis_run(const DevPot &pot, const AxisLane &A, const Ruth4Coef &co, double dt, int64_t n_steps,
                                         int64_t ns, int axis, double &x, double &v, Store store) {
    double g;
    if (!RUTH) {
        // the gradient at x belongs to the start (at = 0) or to step `at`, whose drift is done
        int64_t at = 0;
        double vh = v;
        if constexpr (MODE != 0) {
            if (gradient_axis<MODE>(pot, A, EVEN || ns > 0, x, g)) {
                vh = half_kick(v, g * dt);
                for (;;) {
                    if (++at > n_steps) return;
                    const bool on = EVEN || at <= ns;
                    x = pick(on, x + vh * dt, x);
                    if (!gradient_axis<MODE>(pot, A, on, x, g)) break;
                    const double gd = g * dt;
                    if (SAVE || at == (EVEN ? n_steps : ns)) v = half_kick(vh, gd);
                    vh = pick(on, vh - gd, vh);
                    if (SAVE) store(at);
                }
            }
        }
        for (;;) {
            const double gd = gradient_axis_call(pot, x, axis) * dt;
            if (at == 0) {
                vh = half_kick(v, gd);
            } else {
                if (SAVE || at == (EVEN ? n_steps : ns)) v = half_kick(vh, gd);
                vh = pick(EVEN || at <= ns, vh - gd, vh);
                if (SAVE) store(at);
            }
            if (++at > n_steps) return;
            x = pick(EVEN || at <= ns, x + vh * dt, x);
        }
    } else {
        const bool regular = ordinary(dt) && pot.regular;
        // sub-step 0's zero-weight gradient, as in ruth4_step (the largest coordinate of the orbit)
        auto zero = [&](bool on) {
            unsigned m = (unsigned)__double2hiint(x) & 0x7fffffffu;
            m = max(m, __shfl_xor_sync(0xffffffffu, m, 1));
            m = max(m, __shfl_xor_sync(0xffffffffu, m, 2));
            return __all_sync(0xffffffffu, (regular && m - (923u << 20) < (200u << 20)) || !on);
        };
        int64_t j = 1;
        int s = 0;  // the sub-step to do
        if constexpr (MODE != 0) {
            bool ok = true;
            while (j <= n_steps && ok) {
                const bool on = EVEN || j <= ns;
                if (!zero(on)) break;
                x = pick(on, x + co.c[0] * v * dt, x);
#pragma unroll 1
                for (s = 1; s < 4; s++) {
                    ok = gradient_axis<MODE>(pot, A, on, x, g);
                    if (!ok) break;
                    v = pick(on, v - co.d[s] * g * dt, v);
                    x = pick(on, x + co.c[s] * v * dt, x);
                }
                if (!ok) break;
                s = 0;
                if (SAVE) store(j);
                j++;
            }
        }
        for (; j <= n_steps; j++) {
            const bool on = EVEN || j <= ns;
#pragma unroll 1
            for (; s < 4; s++) {
                if (s > 0 || !zero(on)) {
                    g = gradient_axis_call(pot, x, axis);
                    v = pick(on, v - co.d[s] * g * dt, v);
                }
                x = pick(on, x + co.c[s] * v * dt, x);
            }
            s = 0;
            if (SAVE) store(j);
        }
    }
}

template <int MODE, bool RUTH, bool SAVE_ALL>
__global__ void __launch_bounds__(32) fixed_axis_kernel(const __grid_constant__ DevPot pot, Ruth4Coef co,
                                                        const double *__restrict__ w0, int64_t n,
                                                        const double *__restrict__ t, int64_t ntimes,
                                                        double *__restrict__ out) {
    const int lane = threadIdx.x, c = lane & 3, axis = c < 2 ? c : 2;
    const int64_t orbit = (int64_t)blockIdx.x * 8 + (lane >> 2);
    const bool keep = orbit < n && c < 3;
    const int64_t i = orbit < n ? orbit : n - 1;
    double x = w0[axis * n + i], v = w0[(3 + axis) * n + i];
    double *ox = out + (SAVE_ALL ? axis * ntimes : axis) * n + i;
    double *ov = out + (SAVE_ALL ? (3 + axis) * ntimes : 3 + axis) * n + i;
    auto store = [&](int64_t j) {
        if (keep) {
            __stcs(ox + j * n, x);
            __stcs(ov + j * n, v);
        }
    };
    if (SAVE_ALL) store(0);
    axis_run<MODE, RUTH, true, SAVE_ALL>(pot, axis_lane(pot), co, t[1] - t[0], ntimes - 1, ntimes - 1, axis, x, v, store);
    if (!SAVE_ALL) store(0);
}

template <bool RUTH>
static int launch_axis(const DevPot &dp, const Ruth4Coef &co, const double *w0, int64_t n, const double *t, int64_t ntimes,
                       bool save_all, double *out, cudaStream_t st, const char *name) {
    const unsigned g8 = (unsigned)((n + 7) / 8);
    switch ((axis_mode(dp) << 1) | (save_all ? 1 : 0)) {
#define GX_CASE(m)                                                                                       \
    case 2 * m: fixed_axis_kernel<m, RUTH, false><<<g8, 32, 0, st>>>(dp, co, w0, n, t, ntimes, out); break; \
    case 2 * m + 1: fixed_axis_kernel<m, RUTH, true><<<g8, 32, 0, st>>>(dp, co, w0, n, t, ntimes, out); break
        GX_CASE(0);
        GX_CASE(1);
        GX_CASE(2);
        GX_CASE(3);
#undef GX_CASE
    }
    return check_launch(name);
}

// Whether few enough orbits for one coordinate per lane.
static bool few_orbits(const DevPot &dp, int64_t n) { return !dp.has_scf && !dp.cdev && n <= (int64_t)32 * multiprocessors(); }

// ---------------------------------------------------------------------------
// Batched FP64 form of the same two integrators (the plain form of the batched
// workload): per orbit its own n_steps, dt and integrator, final state only,
// gala's arithmetic exactly as in the kernels above.  Same work queue as the
// FP32 batch kernel (gx_batch.cu, gx_queue.cuh): chunks of the caller's order
// pulled by a persistent grid.
// ---------------------------------------------------------------------------
template <bool SCF>
__global__ void __launch_bounds__(128, 1) batch_fp64_kernel(const __grid_constant__ DevPot pot, Ruth4Coef co,
                                                            int64_t n, int64_t slots, int32_t chunk, int64_t n_lead,
                                                            const double *__restrict__ w0,
                                                            const int64_t *__restrict__ nsteps,
                                                            const double *__restrict__ dtv,
                                                            const int32_t *__restrict__ method,
                                                            const int32_t *__restrict__ order,
                                                            int32_t *__restrict__ counter,
                                                            double *__restrict__ out,
                                                            const int32_t *__restrict__ cancel) {
    const int lane = threadIdx.x & 31;
    const int64_t nchunks = slots / chunk;
    const int subs = chunk / 32;
    int phase = 0;
    for (;;) {
        // a cancelled launch takes no further work (lane 0 decides for the warp)
        int64_t c = -1;
        int sub = -1;
        if (lane == 0 && !cancel_requested(cancel)) c = queue_next(counter, nchunks, n_lead, subs, phase, sub);
        c = __shfl_sync(0xffffffffu, c, 0);
        sub = __shfl_sync(0xffffffffu, sub, 0);
        if (c < 0) break;
        // one lead block, or every block of a main-region chunk
        const int b0 = sub >= 0 ? sub : 0, b1 = sub >= 0 ? sub + 1 : subs;
        for (int b = b0; b < b1; b++) {
            const int32_t i = order[c * chunk + 32 * b + lane];
            // -1 pads the order; any other id outside [0, n) is skipped (and recorded in the debug build)
            if (i == -1 || !GX_DBG_CHECK(i >= 0 && i < n, DBG_ORDER, i, n)) continue;
            GX_DBG_DONE(i, nsteps[i]);
            double w[6], g[3];
            for (int k = 0; k < 6; k++) w[k] = w0[k * n + i];
            const int64_t ns = nsteps[i];
            const double dt = dtv[i];
            if (ns > 0 && method[i] == 0) {
                double vh[3];
                grad(pot, w, g);
                for (int k = 0; k < 3; k++) vh[k] = half_kick(w[3 + k], g[k] * dt);
                for (int64_t j = 0; j < ns; j++) {
                    for (int k = 0; k < 3; k++) w[k] = w[k] + vh[k] * dt;
                    grad(pot, w, g);
                    for (int k = 0; k < 3; k++) {
                        const double gd = g[k] * dt;
                        if (j == ns - 1) w[3 + k] = half_kick(vh[k], gd);
                        vh[k] = vh[k] - gd;
                    }
                }
            } else if (ns > 0) {
                const bool dt_ok = ordinary(dt);
                for (int64_t j = 0; j < ns; j++) ruth4_step<SCF>(pot, co, dt, dt_ok, w);
            }
            for (int k = 0; k < 6; k++) out[k * n + i] = w[k];
        }
    }
}

// The batch with four lanes per orbit: a CTA of four warps takes a 32-orbit block,
// eight orbits to a warp, one CTA per SM.  For batches whose longest orbits set the
// time rather than the FP64 pipe's throughput (batch_lanes): lengths 100 to
// 2,000, MW composite, 16,384 orbits 22.0 ms one lane per orbit, 11.9 ms here; 24,000
// 22.0 and 12.8; 40,001 22.0 and 21.2.  (Four such CTAs per SM: 25.5 ms for 16,384,
// the longest orbits then share their scheduler from the start.)
template <int MODE>
__global__ void __launch_bounds__(128) batch_axis_kernel(const __grid_constant__ DevPot pot, Ruth4Coef co, int64_t n,
                                                         int64_t slots, int32_t chunk, int64_t n_lead,
                                                         const double *__restrict__ w0, const int64_t *__restrict__ nsteps,
                                                         const double *__restrict__ dtv, const int32_t *__restrict__ method,
                                                         const int32_t *__restrict__ order, int32_t *__restrict__ counter,
                                                         double *__restrict__ out, const int32_t *__restrict__ cancel) {
    __shared__ int64_t item;
    __shared__ int item_sub;
    const int lane = threadIdx.x & 31, c = lane & 3, axis = c < 2 ? c : 2;
    const int64_t nchunks = slots / chunk;
    const int subs = chunk / 32;
    const AxisLane A = axis_lane(pot);
    int phase = 0;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) {
            int sub = -1;
            item = cancel_requested(cancel) ? -1 : queue_next_ordered(counter, nchunks, n_lead, subs, phase, sub);
            item_sub = sub;
        }
        __syncthreads();
        const int64_t ch = item;
        const int sub = item_sub;
        if (ch < 0) break;
        const int b0 = sub >= 0 ? sub : 0, b1 = sub >= 0 ? sub + 1 : subs;
        for (int b = b0; b < b1; b++) {
            int32_t i = order[ch * chunk + 32 * b + 8 * (threadIdx.x >> 5) + (lane >> 2)];
            // -1 pads the order; any other id outside [0, n) is skipped (and recorded once in the debug build)
            if (i < 0 || i >= n) {
                if (i != -1 && c == 0) (void)GX_DBG_CHECK(false, DBG_ORDER, i, n);
                i = -1;
            } else if (c == 0) {
                GX_DBG_DONE(i, nsteps[i]);
            }
            // lanes without an orbit go along at a harmless point
            const bool ok = i >= 0;
            double x = ok ? w0[axis * n + i] : 1., v = ok ? w0[(3 + axis) * n + i] : 0.;
            const double dt = ok ? dtv[i] : 0.;
            const int64_t ns = ok ? nsteps[i] : 0;
            auto none = [](int64_t) {};
            // a warp's orbits are of one integrator in the schedule's orders, of both in others
            for (int m = 0; m < 2; m++) {
                const int64_t mine = ok && (method[i] == 0) == (m == 0) && ns > 0 ? ns : 0;
                int64_t most = mine;
                for (int o = 16; o > 0; o >>= 1) {
                    const int64_t other = __shfl_xor_sync(0xffffffffu, most, o);
                    most = other > most ? other : most;
                }
                if (most == 0) continue;
                if (m == 0) axis_run<MODE, false, false, false>(pot, A, co, dt, most, mine, axis, x, v, none);
                else axis_run<MODE, true, false, false>(pot, A, co, dt, most, mine, axis, x, v, none);
            }
            if (ok && c < 3) {
                out[axis * n + i] = x;
                out[(3 + axis) * n + i] = v;
            }
        }
    }
}

// Lanes per orbit of a batch.  An SM takes 32 orbits at a time with four lanes each, and
// one after another beyond that, while one lane per orbit takes 128 at a time: what the
// four lanes gain is a shorter step, and the lengths decide what that is worth.  300
// steps on average, one lane / four, ms:
//   straight run of a composite (0.55 of the step): even Ruth4 lengths 4,864 orbits 3.36
//   / 1.84, 9,800 3.36 / 5.38; spread 20 : 1 17,000 6.61 / 3.59, 24,320 6.60 / 3.92.  The
//   line is where spread lengths still gain (5 : 1 meets there, 20 : 1 at 41,000).
//   one Hernquist sphere (0.45): even Ruth4 9,728 1.86 / 1.61, 14,700 1.86 / 3.12, even
//   Leapfrog 9,728 0.59 / 0.51, 9,800 0.59 / 0.74; 20 : 1 17,000 3.62 / 1.59.  With steps
//   that cheap even lengths are to gain too.
//   component loop (0.83 to 0.9: a lane still evaluates every component): even Ruth4, five
//   to eight components 4,864 0.9, 5,000 1.7 times one lane's; 20 : 1 24,320 0.97.  One
//   block per SM.
static int batch_lanes(const DevPot &dp, int64_t n) {
    if (dp.has_scf || dp.cdev) return 1;
    const int mode = axis_mode(dp);
    const int64_t per_sm = mode == 0 ? 32 : mode == 1 ? 64 : 160;
    return n <= per_sm * multiprocessors() ? 4 : 1;
}

static int fixed_common(const gx_potential *pot, const gx_frame *frame, const double *w0, int64_t n,
                        const double *t, int64_t ntimes, double *w_out, DevPot *dp, const char *name) {
    int rc = pack_potential(pot, dp);
    if (rc) return rc;
    if (frame != nullptr && frame->type != GX_FRAME_STATIC) {
        set_error("%s integration is currently only supported for StaticFrame", name);
        return GX_ERR_UNSUPPORTED;
    }
    GX_CHECK_ARG(n >= 0, "n < 0");
    GX_CHECK_ARG(ntimes >= 2, "ntimes must be >= 2 (got %lld)", (long long)ntimes);
    GX_CHECK_ARG(n == 0 || (w0 && t && w_out), "NULL array");
    return GX_OK;
}

}  // namespace gx

extern "C" {

int gx_leapfrog_integrate_hamiltonian(const gx_potential *pot, const gx_frame *frame, const double *w0, int64_t n,
                                      const double *t, int64_t ntimes, int32_t save_all, double *w_out,
                                      void *stream) {
    gx::DevPot dp;
    int rc = gx::fixed_common(pot, frame, w0, n, t, ntimes, w_out, &dp, "Leapfrog");
    if (rc || n == 0) return rc;
    const int bs = 128;
    const unsigned grid = (unsigned)((n + bs - 1) / bs);
    cudaStream_t st = gx::as_stream(stream);
    if (gx::few_orbits(dp, n))
        return gx::launch_axis<false>(dp, gx::Ruth4Coef{}, w0, n, t, ntimes, save_all, w_out, st, "leapfrog");
    if (save_all && dp.has_scf)
        gx::leapfrog_kernel<true, true><<<grid, bs, 0, st>>>(dp, w0, n, t, ntimes, w_out);
    else if (save_all)
        gx::leapfrog_kernel<true, false><<<grid, bs, 0, st>>>(dp, w0, n, t, ntimes, w_out);
    else if (dp.has_scf)
        gx::leapfrog_kernel<false, true><<<grid, bs, 0, st>>>(dp, w0, n, t, ntimes, w_out);
    else
        gx::leapfrog_kernel<false, false><<<grid, bs, 0, st>>>(dp, w0, n, t, ntimes, w_out);
    return gx::check_launch("leapfrog");
}

int gx_batch_integrate_fp64(const gx_potential *pot, const double *w0, int64_t n, const int64_t *n_steps,
                            const double *dt, const int32_t *method, const int32_t *order, int64_t n_slots,
                            int32_t chunk, int32_t block, int32_t grid, int32_t *queue_counter, double *w_out,
                            void *stream) {
    gx::DevPot dp;
    int rc = gx::pack_potential(pot, &dp);
    if (rc) return rc;
    GX_CHECK_ARG(n >= 0 && n < (int64_t)INT32_MAX, "n out of range");
    if (n == 0) return GX_OK;
    GX_CHECK_ARG(w0 && n_steps && dt && method && order && queue_counter && w_out, "NULL array");
    GX_CHECK_ARG(chunk >= 32 && chunk % 32 == 0 && chunk <= 4096, "chunk must be a multiple of 32 in [32, 4096]");
    GX_CHECK_ARG(n_slots >= n && n_slots % chunk == 0, "order length must be >= n and a multiple of chunk");
    GX_CHECK_ARG(block >= 32 && block <= 128 && block % 32 == 0, "block must be a multiple of 32 in [32, 128]");
    GX_CHECK_ARG(grid >= 1, "grid must be >= 1");
    const double two_13 = std::pow(2., 1. / 3.);
    gx::Ruth4Coef co;
    co.c[0] = 1. / (2. * (2. - two_13));
    co.c[1] = (1. - two_13) / (2. * (2. - two_13));
    co.c[2] = (1. - two_13) / (2. * (2. - two_13));
    co.c[3] = 1. / (2. * (2. - two_13));
    co.d[0] = 0.;
    co.d[1] = 1. / (2. - two_13);
    co.d[2] = -two_13 / (2. - two_13);
    co.d[3] = 1. / (2. - two_13);
    cudaStream_t st = gx::as_stream(stream);
    GX_CUDA_TRY(cudaMemsetAsync(queue_counter, 0, GX_BATCH_QUEUE_WORDS * sizeof(int32_t), st));
    const int64_t n_lead = gx::queue_lead_chunks(n_slots / chunk, chunk);
    if (gx::batch_lanes(dp, n) == 4) {
        const auto kernel = gx::axis_mode(dp) == 0   ? gx::batch_axis_kernel<0>
                            : gx::axis_mode(dp) == 1 ? gx::batch_axis_kernel<1>
                            : gx::axis_mode(dp) == 2 ? gx::batch_axis_kernel<2>
                                                     : gx::batch_axis_kernel<3>;
        // one CTA per SM, one warp per scheduler: the longest orbits, which go first, keep their pace
        const int sms = gx::multiprocessors();
        kernel<<<sms > 0 && sms < grid ? sms : grid, 128, 0, st>>>(dp, co, n, n_slots, chunk, n_lead, w0, n_steps, dt, method, order, queue_counter, w_out,
                                     gx::cancel_flag());
    }
    else if (dp.has_scf)
        gx::batch_fp64_kernel<true><<<grid, block, 0, st>>>(dp, co, n, n_slots, chunk, n_lead, w0, n_steps, dt,
                                                            method, order, queue_counter, w_out, gx::cancel_flag());
    else
        gx::batch_fp64_kernel<false><<<grid, block, 0, st>>>(dp, co, n, n_slots, chunk, n_lead, w0, n_steps, dt,
                                                             method, order, queue_counter, w_out, gx::cancel_flag());
    return gx::check_launch("batch_fp64");
}

int gx_batch_fp64_lanes(const gx_potential *pot, int64_t n, int32_t *lanes) {
    gx::DevPot dp;
    int rc = gx::pack_potential(pot, &dp);
    if (rc) return rc;
    GX_CHECK_ARG(n >= 0, "n < 0");
    GX_CHECK_ARG(lanes, "NULL pointer");
    *lanes = gx::batch_lanes(dp, n);
    return GX_OK;
}

int gx_ruth4_integrate_hamiltonian(const gx_potential *pot, const gx_frame *frame, const double *w0, int64_t n,
                                   const double *t, int64_t ntimes, int32_t save_all, double *w_out,
                                   void *stream) {
    gx::DevPot dp;
    int rc = gx::fixed_common(pot, frame, w0, n, t, ntimes, w_out, &dp, "Ruth4");
    if (rc || n == 0) return rc;
    // ruth4.pyx:65-78, evaluated on the host in double like Cython does.
    const double two_13 = std::pow(2., 1. / 3.);
    gx::Ruth4Coef co;
    co.c[0] = 1. / (2. * (2. - two_13));
    co.c[1] = (1. - two_13) / (2. * (2. - two_13));
    co.c[2] = (1. - two_13) / (2. * (2. - two_13));
    co.c[3] = 1. / (2. * (2. - two_13));
    co.d[0] = 0.;
    co.d[1] = 1. / (2. - two_13);
    co.d[2] = -two_13 / (2. - two_13);
    co.d[3] = 1. / (2. - two_13);
    const int bs = 128;
    const unsigned grid = (unsigned)((n + bs - 1) / bs);
    cudaStream_t st = gx::as_stream(stream);
    if (gx::few_orbits(dp, n)) return gx::launch_axis<true>(dp, co, w0, n, t, ntimes, save_all, w_out, st, "ruth4");
    if (save_all && dp.has_scf)
        gx::ruth4_kernel<true, true><<<grid, bs, 0, st>>>(dp, co, w0, n, t, ntimes, w_out);
    else if (save_all)
        gx::ruth4_kernel<true, false><<<grid, bs, 0, st>>>(dp, co, w0, n, t, ntimes, w_out);
    else if (dp.has_scf)
        gx::ruth4_kernel<false, true><<<grid, bs, 0, st>>>(dp, co, w0, n, t, ntimes, w_out);
    else
        gx::ruth4_kernel<false, false><<<grid, bs, 0, st>>>(dp, co, w0, n, t, ntimes, w_out);
    return gx::check_launch("ruth4");
}

}  // extern "C"
