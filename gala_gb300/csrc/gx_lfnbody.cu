// gx_lfnbody.cu -- FP64 Leapfrog for small direct n-body systems and for the
// release systems of Leapfrog mock streams (gala's arithmetic, -fmad=false).
#include "gx_host.h"
#include "gx_scf.cuh"
#include "gx_body.cuh"

namespace gx {

// ---------------------------------------------------------------------------
// Leapfrog n-body systems: leapfrog_integrate_nbody (leapfrog.pyx:161-255) and
// the release systems of mockstream_leapfrog (mockstream.pyx:548-593).  gala moves
// the bodies in order within a step: body k drifts, feels the external potential
// and every other non-null massive body at its CURRENT position (already moved this
// step when j < k: c_nbody_gradient_symplectic, cpotential.cpp:418-442), and kicks.
// A drift depends on nothing but the body itself, so a system is a GROUP of lanes,
// one per body: all drift, and body k takes body j's position after the drift
// (j < k) or before it (j > k) from its lane.  The same operations in the same
// order as one thread per system, with a step as long as one body's instead of the
// sum over them: the kernel was bound by those chains (5 warps per SM and about 330
// FP64 instructions per step), now by the FP64 pipe (16 warps, 115 instructions;
// the release systems of 64 streams x 400 releases take 4.6 ms; the whole call 20.3 -> 13.0 ms).
// Consecutive groups are consecutive systems of one release time, so a warp runs
// systems of equal length; one-warp CTAs, longest first, fill the SMs evenly.
// ---------------------------------------------------------------------------
struct LfArgs {
    int64_t n_sys;
    int32_t nbody;          // massive bodies (first in every system)
    int32_t nparticles;     // direct n-body: bodies per system
    const gx_body *bodies;  // (n_streams or n_sys, nbody)
    double dt;
    // direct n-body systems
    const double *w0;       // (n_sys, nparticles, 6)
    const double *t;
    int64_t ntimes;
    int32_t save_all;
    double *w_out;
    // release systems
    int64_t n_streams, n_release, n_particles;
    const double *nbody_w;  // (n_streams, n_release, nbody, 6)
    const double *release_t;
    const int64_t *offset;
    const double *stream_w0;
    double t_final;
    double *stream_w_out, *nbody_w_out;
    int32_t *status;
    int32_t gs;             // lanes per group (the largest system)
    // release systems larger than max_per_release said go in a launch of their own:
    int32_t upto;           // systems of more members than this get status -1
    int32_t over;           // > 0: only systems of more members than this are this launch's
};

// Gradient at the lane's body, x after this step's drift and xo before it.  All 32
// lanes take part: shuffles within a group's own mask would each wait on a
// synchronisation.
template <bool SCF>
__device__ __forceinline__ void lf_grad(const DevPot &pot, int base, int member, bool in_sys, int nbody,
                                        const gx_body *__restrict__ bod, const double *xo, const double *x, double *g) {
    V3 q;
    for (int k = 0; k < 3; k++) q.v[k] = x[k];
    const V3 ge = gradient_call<SCF, true>(pot, q);
    for (int k = 0; k < 3; k++) g[k] = ge.v[k];
    for (int j = 0; j < nbody; j++) {
        double d[3];
        for (int k = 0; k < 3; k++) {
            const double xn = __shfl_sync(0xffffffffu, x[k], base + j), xp = __shfl_sync(0xffffffffu, xo[k], base + j);
            d[k] = x[k] - (j < member ? xn : xp);
        }
        const int type = __ldg(&bod[j].type);
        if (!in_sys || j == member || type == GX_POT_NULL) continue;
        const V3 f2 = body_gradient_call<true>(type, bod[j].params, d[0], d[1], d[2]);
        for (int k = 0; k < 3; k++) g[k] += f2.v[k];
    }
}

template <bool STREAM, bool SAVE_ALL, bool SCF>
__global__ void __launch_bounds__(32) lf_nbody_kernel(const __grid_constant__ DevPot pot, const LfArgs A) {
    const int gs = A.gs, lane = threadIdx.x;
    const int grp = lane / gs, member = lane - grp * gs, base = grp * gs;
    const int64_t sys = (int64_t)blockIdx.x * (32 / gs) + grp;
    const double dt = A.dt;
    // a lane without a system or a body goes along at a harmless point
    bool in_sys = grp < 32 / gs && sys < A.n_sys;
    const gx_body *bod = A.bodies;
    int64_t si = 0, ss = 0, n_steps = 0;
    const double *src = nullptr;
    double *o = nullptr;  // where the lane's body goes
    int32_t *done = nullptr;
    if (in_sys) {
        if constexpr (STREAM) {
            si = sys / A.n_streams;
            ss = sys - si * A.n_streams;
            const int64_t o0 = A.offset[si], o1 = A.offset[si + 1];
            const int64_t size = A.nbody + (o1 - o0);
            const bool rows = o1 >= o0 && o0 >= 0 && o1 <= A.n_particles;
            const bool bad = !A.over && (!rows || size > A.upto);
            const bool here = rows && o1 > o0 && size > A.over && size <= gs;
            if (member == 0) {
                int32_t *const status = A.status + ss * A.n_release + si;
                if (bad) (void)GX_DBG_CHECK(!bad, DBG_OFFSET, si, A.n_release);
                if (bad || (!A.over && o1 == o0)) *status = bad ? -1 : 0;
                if (here) done = status;
            }
            bod = A.bodies + ss * A.nbody;
            in_sys = here && member < (int)size;
            if (in_sys) {
                n_steps = (int64_t)((A.t_final - A.release_t[si]) / dt + 0.5);  // mockstream.pyx:582
                if (member < A.nbody) {
                    src = A.nbody_w + ((ss * A.n_release + si) * A.nbody + member) * 6;
                    if (A.nbody_w_out && o1 == A.offset[A.n_release]) o = A.nbody_w_out + (ss * A.nbody + member) * 6;
                } else {
                    const int64_t row = ss * A.n_particles + o0 + (member - A.nbody);
                    src = A.stream_w0 + row * 6;
                    o = A.stream_w_out + row * 6;
                }
            }
        } else {
            bod = A.bodies + sys * A.nbody;
            in_sys = member < A.nparticles;
            if (in_sys) {
                n_steps = A.ntimes - 1;
                src = A.w0 + (sys * A.nparticles + member) * 6;
                o = A.w_out + ((SAVE_ALL ? sys * A.ntimes : sys) * A.nparticles + member) * 6;
            }
        }
    }
    if (STREAM && A.over && !__any_sync(0xffffffffu, in_sys)) return;
    int64_t most = n_steps;  // the warp's longest system
    for (int k = 16; k > 0; k >>= 1) {
        const int64_t other = __shfl_xor_sync(0xffffffffu, most, k);
        most = other > most ? other : most;
    }
    double x[3], v[3], vh[3], xo[3], g[3];
    for (int k = 0; k < 3; k++) {
        x[k] = in_sys ? src[k] : 1.;
        v[k] = in_sys ? src[3 + k] : 0.;
    }
    auto store = [&](double *p) {
        for (int k = 0; k < 3; k++) {
            p[k] = x[k];
            p[3 + k] = v[k];
        }
    };
    if (SAVE_ALL && o) store(o);
    // c_init_velocity_nbody (leapfrog.pyx:126-138), every body at the start positions
    lf_grad<SCF>(pot, base, member, in_sys, A.nbody, bod, x, x, g);
    for (int k = 0; k < 3; k++) vh[k] = fma(-0.5, g[k] * dt, v[k]);  // v - g * dt / 2., the halving exact
    for (int64_t j = 0; j < most; j++) {
        const bool on = j < n_steps;
        // c_leapfrog_step_nbody (leapfrog.pyx:140-158)
        for (int k = 0; k < 3; k++) {
            xo[k] = x[k];
            x[k] = pick(on, x[k] + vh[k] * dt, x[k]);
        }
        lf_grad<SCF>(pot, base, member, in_sys, A.nbody, bod, xo, x, g);
        for (int k = 0; k < 3; k++) {
            const double gd = g[k] * dt;
            if (on && (SAVE_ALL || j == n_steps - 1)) v[k] = fma(-0.5, gd, vh[k]);
            vh[k] = pick(on, vh[k] - gd, vh[k]);
        }
        if (SAVE_ALL && o && on) store(o + (j + 1) * A.nparticles * 6);
    }
    if (!SAVE_ALL && o) store(o);
    if (STREAM && done) *done = 1;
}

template <bool STREAM, bool SAVE_ALL>
int launch_lf(const DevPot &dp, LfArgs A, int members, cudaStream_t st) {
    if (members > 8) {
        set_error("leapfrog n-body systems of %d bodies: at most 8", members);
        return GX_ERR_UNSUPPORTED;
    }
    // max_per_release sizes the groups; releases beyond it, up to three or eight
    // members, are taken all the same, by groups of that size
    const int most = dp.has_scf || members > 3 ? 8 : 3;
    A.upto = most;
    for (A.gs = members;; A.gs = most) {
        const int64_t per = 32 / A.gs;
        const unsigned grid = (unsigned)((A.n_sys + per - 1) / per);
        if (dp.has_scf)
            lf_nbody_kernel<STREAM, SAVE_ALL, true><<<grid, 32, 0, st>>>(dp, A);
        else
            lf_nbody_kernel<STREAM, SAVE_ALL, false><<<grid, 32, 0, st>>>(dp, A);
        if (!STREAM || A.gs == most) break;
        A.over = members;
    }
    return check_launch(STREAM ? "mockstream_leapfrog" : "nbody_leapfrog");
}

}  // namespace gx

extern "C" int gx_nbody_leapfrog(const gx_potential *pot, int64_t n_systems, int32_t nparticles, int32_t nbody,
                                 const gx_body *bodies, const double *w0, const double *t, int64_t ntimes,
                                 int32_t save_all, double *w_out, void *stream) {
    gx::DevPot dp;
    int rc = gx::pack_potential(pot, &dp);
    if (rc) return rc;
    GX_CHECK_ARG(n_systems >= 0, "n_systems < 0");
    GX_CHECK_ARG(nparticles >= 1 && nparticles <= 8, "nparticles must be in [1, 8] (got %d)", nparticles);
    GX_CHECK_ARG(nbody >= 0 && nbody <= nparticles, "nbody must be in [0, nparticles] (got %d)", nbody);
    GX_CHECK_ARG(ntimes >= 2, "ntimes must be >= 2 (got %lld)", (long long)ntimes);
    if (n_systems == 0) return GX_OK;
    GX_CHECK_ARG(w0 && t && w_out, "NULL array");
    GX_CHECK_ARG(nbody == 0 || bodies, "bodies is NULL");
    double t01[2];
    GX_CUDA_TRY(cudaMemcpyAsync(t01, t, sizeof(t01), cudaMemcpyDeviceToHost, gx::as_stream(stream)));
    GX_CUDA_TRY(cudaStreamSynchronize(gx::as_stream(stream)));
    gx::LfArgs A;
    memset(&A, 0, sizeof(A));
    A.n_sys = n_systems;
    A.nbody = nbody;
    A.nparticles = nparticles;
    A.bodies = bodies;
    A.dt = t01[1] - t01[0];
    A.w0 = w0;
    A.t = t;
    A.ntimes = ntimes;
    A.save_all = save_all ? 1 : 0;
    A.w_out = w_out;
    cudaStream_t st = gx::as_stream(stream);
    return save_all ? gx::launch_lf<false, true>(dp, A, nparticles, st)
                    : gx::launch_lf<false, false>(dp, A, nparticles, st);
}

extern "C" int gx_mockstream_leapfrog(const gx_potential *pot, int64_t n_streams, int32_t nbody,
                                      const gx_body *bodies, const double *nbody_w, int64_t n_release,
                                      const double *release_t, const int64_t *release_offset,
                                      int32_t max_per_release, const double *stream_w0, int64_t n_particles,
                                      double t_final, double dt, double *stream_w_out, double *nbody_w_out,
                                      int32_t *status, void *stream) {
    gx::DevPot dp;
    int rc = gx::pack_potential(pot, &dp);
    if (rc) return rc;
    GX_CHECK_ARG(n_streams >= 0 && n_release >= 0 && n_particles >= 0, "negative size");
    GX_CHECK_ARG(nbody >= 1, "nbody must be >= 1 (the progenitor)");
    GX_CHECK_ARG(max_per_release >= 0 && nbody + max_per_release <= 8,
                 "nbody + max_per_release must be <= 8 (got %d + %d)", nbody, max_per_release);
    GX_CHECK_ARG(dt != 0.0, "dt must be non-zero");
    if (n_streams == 0 || n_release == 0) return GX_OK;
    GX_CHECK_ARG(bodies && nbody_w && release_t && release_offset && status, "NULL array");
    GX_CHECK_ARG(n_particles == 0 || (stream_w0 && stream_w_out), "NULL particle array");
    gx::LfArgs A;
    memset(&A, 0, sizeof(A));
    A.n_sys = n_streams * n_release;
    A.nbody = nbody;
    A.bodies = bodies;
    A.dt = dt;
    A.n_streams = n_streams;
    A.n_release = n_release;
    A.n_particles = n_particles;
    A.nbody_w = nbody_w;
    A.release_t = release_t;
    A.offset = release_offset;
    A.stream_w0 = stream_w0;
    A.t_final = t_final;
    A.stream_w_out = stream_w_out;
    A.nbody_w_out = nbody_w_out;
    A.status = status;
    return gx::launch_lf<true, false>(dp, A, nbody + max_per_release, gx::as_stream(stream));
}
