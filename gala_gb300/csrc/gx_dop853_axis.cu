// gx_dop853_axis.cu -- FP64 DOP853 for few orbits: four lanes per orbit, one
// coordinate each (position and momentum; the fourth lane repeats z).
//
// The arithmetic, the batch semantics and the step control are those of
// gx_dop853.cu.  What differs is what bounds them: an FP64 instruction costs a warp 64
// cycles whatever its lanes do, and a few batches of orbits leave most of the 608
// schedulers idle, so the coordinates go side by side: a step takes about 500
// FP64 instructions instead of 823 (static frame) or 1,500 (rotating frame).  37
// orbits through a rotating bar, 400 Myr, every Myr kept: 59 -> 18 ms (one lane per orbit / here).
//   * A batch is a cluster of up to 8 CTAs of 1, 2 or 4 warps, 8 orbits to a warp
//     (100 orbits: 7 CTAs of 2 warps), spread over as many SMs.
//   * The right-hand side gathers the point by shuffles, and each lane evaluates one of
//     up to four components: every closed form is a root, a root or reciprocal or
//     logarithm of something made from it, and a factor times the position, so the
//     four types go through one straight run with the lane's constants (AxisComp),
//     and three additions bring the factors together.
//   * The step's sums: a warp fold, one store per CTA of the cluster through
//     distributed shared memory, one cluster barrier, and the same fold over the
//     warps' partial sums in every warp, so all decide alike.
// Frames: static, and rotating at a constant rate (cross products from the
// neighbours' lanes).  Closed-form components in the by-value descriptor.
#include "gx_dop853.cuh"
#include "gx_dop853_tableau.cuh"
#include "gx_fast64.cuh"

namespace gx {

constexpr int AXIS_MAX_WARPS = 32;  // of a batch

struct V2 {
    double x, v;
};

namespace fast {

// The lane's component of the gradient at the group's point.
static __device__ __noinline__ double gradient_axis_general(const DevPot &pot, double q, int axis) {
    const double p[3] = {quad(q, 0), quad(q, 1), quad(q, 2)};
    Diag d;
    d.init(p);
    double gs = 0.;
    for (int i = 0; i < pot.ncomp; i++) {
        const DevComp &c = pot.c[i];
        if (c.do_sr == 0) {
            comp_gradient_f(pot, i, p, d);
        } else {
            double qt[3], gt[3];
            shift_rotate(c, p, qt);
            Diag dt;
            dt.init(qt);
            comp_gradient_f(pot, i, qt, dt);
            dt.gradient(qt, gt);
            gs += fma(c.R[axis], gt[0], fma(c.R[3 + axis], gt[1], c.R[6 + axis] * gt[2]));
        }
    }
    return fma(d.F + (axis == 0 ? d.A[0] : axis == 1 ? d.A[1] : d.A[2]), q, gs);
}

// A component as the lane that evaluates it needs it: m^2 = k0 x^2 + k1 y^2 + k2 z^2 + k3,
// s = sqrt(m^2), den = e1 s + e0 (Hernquist s + c, NFW 1 + u), and the factor
// G m i p^2 X along (w0, w1, w2) with i = 1 / s, p = i, X = 1 but where the type says
// otherwise.
struct AxisComp {
    double gm, k0, k1, k2, k3, e0, e1, irs, a, w0, w1, w2;
    int type;
};

__device__ __forceinline__ AxisComp axis_comp(const DevPot &pot, int i) {
    AxisComp L = {0., 1., 1., 1., 1., 1., 0., 0., 0., 1., 1., 1., GX_POT_NULL};  // adds nothing
    if (i >= pot.ncomp) return L;
    const DevComp &C = pot.c[i];
    if (C.type == GX_POT_NULL) return L;
    L.type = C.type;
    L.gm = C.dc[0];
    L.k3 = 0.;
    if (C.type == GX_POT_HERNQUIST) {
        L.e1 = 1.;
        L.e0 = pot.p[C.poff + 2];
    } else if (C.type == GX_POT_PLUMMER) {
        L.k3 = C.dc[1];
    } else if (C.type == GX_POT_MIYAMOTONAGAI) {
        L.k0 = L.k1 = 0.;
        L.k3 = C.dc[1];
        L.a = pot.p[C.poff + 2];
    } else if (C.type != GX_POT_KEPLER) {  // the NFW shapes
        L.e1 = L.irs = C.dc[1];
        if (C.type != GX_POT_SPHERICALNFW) {
            L.k0 = L.w0 = C.dc[2];
            L.k1 = L.w1 = C.dc[3];
            L.k2 = L.w2 = C.dc[4];
        }
    }
    return L;
}

// The lane's component of the gradient, one potential component per lane.  False, for
// the whole warp, where an argument is outside the integer forms' range.
__device__ __forceinline__ bool gradient_axis_lanes(const AxisComp *tab, double q, double &g) {
    const int c = threadIdx.x & 3;
    const AxisComp &L = tab[c];
    const int type = L.type;
    const bool mn = type == GX_POT_MIYAMOTONAGAI, hern = type == GX_POT_HERNQUIST;
    const bool nfw = type == GX_POT_SPHERICALNFW || type == GX_POT_FLATTENEDNFW || type == GX_POT_TRIAXIALNFW;
    const double x = quad(q, 0), y = quad(q, 1), z = quad(q, 2);
    const double xy2 = fma(x, x, y * y);
    const double m2 = fma(L.k0 * x, x, fma(L.k1 * y, y, fma(L.k2 * z, z, L.k3)));
    double is;
    const double s = ip::sqrt_rsqrt_u(m2, is);
    const double den = fma(s, L.e1, L.e0), u = s * L.irs;
    const double zd = L.a + s;
    const double W = fma(zd, zd, xy2);
    const double rc = ip::rcp_u(den);
    const double iW = ip::rsqrt_u(W);
    const double ln = ip::ln_n(den);
    const bool ok = ip::ok_sqrt(m2) & ip::ok_rcp(den) & (!mn | ip::ok_sqrt(W)) & (!nfw | ip::ln_range(den));
    const double X = pick(nfw, fma(-u, rc, ln), 1.0);
    const double i = pick(mn, iW, is), p = pick(hern, rc, i);
    const double f = (L.gm * i) * (p * p) * X;
    const double fx = f * L.w0, fy = f * L.w1, fz = f * pick(mn, fma(L.a, is, 1.0), L.w2);
    // lane 0 collects x, lane 1 y, lanes 2 and 3 z
    const bool xy = c < 2;
    const double r1 = __shfl_xor_sync(0xffffffffu, pick(xy, fz, fx), 2), r2 = __shfl_xor_sync(0xffffffffu, fy, 2);
    const double v1 = pick(xy, fx, fz) + r1, v2 = fy + r2;
    const double r3 = __shfl_xor_sync(0xffffffffu, pick(c == 0, v2, v1), 1);
    g = (pick(c == 1, v2, v1) + r3) * q;
    return __all_sync(0xffffffffu, ok);
}

// Hamilton's equations for the lane's coordinate (rhs_call_f in gx_fast64.cuh).
template <bool LANES, bool ROT>
static __device__ __noinline__ V2 axis_rhs(const DevPot &pot, const DevFrame &fr, const AxisComp *tab, double q, double p) {
    const int c = threadIdx.x & 3, axis = c < 2 ? c : 2;
    double g;
    if (!LANES || !gradient_axis_lanes(tab, q, g)) g = gradient_axis_general(pot, q, axis);
    V2 f;
    if (ROT) {
        const int a = axis == 2 ? 0 : axis + 1, b = axis == 0 ? 2 : axis - 1;  // the next two axes
        const double Oa = fr.O[a], Ob = fr.O[b];
        const double qa = __shfl_sync(0xffffffffu, q, a, 4), qb = __shfl_sync(0xffffffffu, q, b, 4);
        const double pa = __shfl_sync(0xffffffffu, p, a, 4), pb = __shfl_sync(0xffffffffu, p, b, 4);
        f.x = p - fma(Oa, qb, -Ob * qa);
        f.v = -(g + fma(Oa, pb, -Ob * pa));
    } else {
        f.x = p;
        f.v = -g;
    }
    return f;
}

}  // namespace fast

// Folds a (lower half) and b (upper half) over a warp: lane 0 holds the sum of a, lane 16 that of b.
__device__ __forceinline__ double fold2(double a, double b) {
    const bool low = (threadIdx.x & 16) == 0;
    const double oa = __shfl_xor_sync(0xffffffffu, a, 16), ob = __shfl_xor_sync(0xffffffffu, b, 16);
    double v = pick(low, a, b) + pick(low, oa, ob);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

struct AxisBatch {
    int G, W, T;        // CTAs, warps per CTA, warps
    unsigned rank, wi;  // CTA, warp of the batch
};

// Batch-wide sums, the same bits in every lane of every warp; buf: one of two used in turn.
__device__ __forceinline__ void axis_sum2(double &a, double &b, double (*buf)[AXIS_MAX_WARPS], const AxisBatch &B) {
    const int lane = threadIdx.x & 31;
    double v = fold2(a, b);
    if (B.T > 1) {
        if ((lane & 15) < B.G) cluster_store(&buf[lane >> 4][B.wi], lane & 15, v);
        cluster_sync_all();
        v = fold2(lane < B.T ? buf[0][lane] : 0., lane < B.T ? buf[1][lane] : 0.);
    }
    a = __shfl_sync(0xffffffffu, v, 0);
    b = __shfl_sync(0xffffffffu, v, 16);
}

#define RHS(xin, vin, kx, kv)                                                \
    do {                                                                     \
        const V2 r_ = fast::axis_rhs<LANES, ROT>(pot, fr, tab, (xin), (vin)); \
        kx = r_.x;                                                           \
        kv = r_.v;                                                           \
    } while (0)

template <bool LANES, bool ROT>
__global__ void __launch_bounds__(128)
dop853_axis_kernel(const __grid_constant__ DevPot pot, const __grid_constant__ DevFrame fr, DopArgs A, int G,
                   const double *__restrict__ w0, int64_t n, const double *__restrict__ t, double *__restrict__ out,
                   int32_t *__restrict__ status, int64_t *__restrict__ stats) {
    using namespace dop;
    __shared__ double buf[2][2][AXIS_MAX_WARPS];
    __shared__ fast::AxisComp tab[4];
    __shared__ int stop;
    if (LANES && threadIdx.x < 4) tab[threadIdx.x] = fast::axis_comp(pot, threadIdx.x);
    AxisBatch B;
    B.G = G;
    B.W = blockDim.x >> 5;
    B.T = G * B.W;
    B.rank = G == 1 ? 0u : cluster_rank();
    const int lane = threadIdx.x & 31, c = lane & 3, axis = c < 2 ? c : 2;
    B.wi = B.rank * B.W + (threadIdx.x >> 5);
    // a batch that starts after cancellation is not integrated: the cluster takes
    // the decision of its first warp
    if (B.T == 1) {
        if (lane == 0) stop = cancel_requested(A.cancel);
        __syncwarp();
    } else {
        cluster_sync_all();  // every CTA's shared memory exists
        if (B.wi == 0) {
            double s = 0.;
            if (lane == 0) s = cancel_requested(A.cancel) ? 1. : 0.;
            s = __shfl_sync(0xffffffffu, s, 0);
            if (lane < G) cluster_store(&buf[0][0][0], lane, s);
        }
        cluster_sync_all();
        if (threadIdx.x == 0) stop = buf[0][0][0] != 0.;
        cluster_sync_all();
    }
    if (stop) return;
    __syncthreads();

    const int64_t b = blockIdx.x / G;
    const int64_t i0 = b * A.nbatch;
    const int nb = (int)min((int64_t)A.nbatch, n - i0);
    const int j = (int)B.wi * 8 + (lane >> 2);
    const bool active = j < nb && c < 3;  // a coordinate of an orbit of the batch
    const double nsys = 6 * nb;

    // lanes without an orbit go along with the batch's last one and add nothing to the sums: an
    // orbit of their own would choose between the forms of the force for the real ones in its warp
    const int jw = min(j, nb - 1);
    double x = w0[axis * n + i0 + jw], v = w0[(3 + axis) * n + i0 + jw];
    double x1, x2, x3, x4, x5, x6, x7, x8, x9, x10, v1, v2, v3, v4, v5, v6, v7, v8, v9, v10, xs, vs, xn, vn;

    // dop853() front-end defaults with dop853_helper's arguments (dop853.pyx:157-182)
    double tx = t[0];
    const double xend = t[A.ntimes - 1];
    double h = t[1] - t[0];
    double hmax = A.dt_max;
    const double uround = 2.220446049250313e-16;
    const double safe = 0.9, fac1 = 0.333, fac2 = 6.0;  // and beta = 0
    int64_t nmax = A.nmax, nstiff = A.nstiff;
    if (!nmax) nmax = 1000000;
    if (!nstiff) nstiff = 1000;
    else if (nstiff < 0) nstiff = nmax + 10;
    if (hmax == 0.0) hmax = xend - tx;
    const double facc1 = 1.0 / fac1, facc2 = 1.0 / fac2;
    const double posneg = sign_d(1.0, xend - tx);
    const double atoli = A.atol, rtoli = A.rtol;
    int last = 0, reject = 0, iasti = 0, nonsti = 0, idid = 0, par = 0;
    double hlamb = 0.0;
    int64_t nfcn = 0, nstep = 0, naccpt = 0, nrejct = 0;
    int64_t out_idx = 0, out_slot = 0, kept = 0;  // kept: the next time of the grid that is stored
    int64_t to_test = nstiff;                     // accepted steps until the next stiffness test

    RHS(x, v, x1, v1);
    hmax = fabs(hmax);
    if (h == 0.0) {
        // hinit (dop853.cpp:18-86), scalar tolerances, batch-wide norms
        const double skx = atoli + rtoli * fabs(x), skv = atoli + rtoli * fabs(v);
        double q = ddiv(x1, skx), p = ddiv(v1, skv);
        double dnf = active ? q * q + p * p : 0.;
        q = ddiv(x, skx);
        p = ddiv(v, skv);
        double dny = active ? q * q + p * p : 0.;
        axis_sum2(dnf, dny, buf[par], B);
        par ^= 1;
        double hh = ((dnf <= 1.0E-10) || (dny <= 1.0E-10)) ? 1.0E-6 : sqrt(dny / dnf) * 0.01;
        hh = min_d(hh, hmax);
        hh = sign_d(hh, posneg);
        RHS(x + hh * x1, v + hh * v1, x2, v2);
        q = ddiv(x2 - x1, skx);
        p = ddiv(v2 - v1, skv);
        double der2 = active ? q * q + p * p : 0., unused = 0.0;
        axis_sum2(der2, unused, buf[par], B);
        par ^= 1;
        der2 = sqrt(der2) / hh;
        const double der12 = max_d(fabs(der2), sqrt(dnf));
        const double h1 = (der12 <= 1.0E-15) ? max_d(1.0E-6, fabs(hh) * 1.0E-3) : pow(0.01 / der12, 1.0 / 8.0);
        hh = min_d(100.0 * fabs(hh), min_d(h1, hmax));
        h = sign_d(hh, posneg);
    }
    nfcn += 2;

    // every scalar below is the same in all warps of the batch
    for (;;) {
        if (h != h) nan_steps(nmax, naccpt, nstep, nfcn, nrejct);
        if (nstep > nmax) {
            idid = -2;
            break;
        }
        if (0.1 * fabs(h) <= fabs(tx) * uround) {
            idid = -3;
            break;
        }
        if ((tx + 1.01 * h - xend) * posneg > 0.0) {
            h = xend - tx;
            last = 1;
        }
        const double xold = tx, hout = h;
        nstep++;

        // the twelve stages (dop853.cpp:368-414), for the position and the momentum
#define STAGE(expr)            \
    do {                       \
        {                      \
            GX_K(x)            \
            xs = fma(h, expr, x); \
        }                      \
        {                      \
            GX_K(v)            \
            vs = fma(h, expr, v); \
        }                      \
    } while (0)
#define GX_K(p)                                                                                                    \
    const double k1 = p##1, k2 = p##2, k3 = p##3, k4 = p##4, k5 = p##5, k6 = p##6, k7 = p##7, k8 = p##8, k9 = p##9, \
                 k10 = p##10;                                                                                      \
    (void)k1, (void)k2, (void)k3, (void)k4, (void)k5, (void)k6, (void)k7, (void)k8, (void)k9, (void)k10;
        xs = fma(h * a21, x1, x);
        vs = fma(h * a21, v1, v);
        RHS(xs, vs, x2, v2);
        xs = fma(h, fma(a32, x2, a31 * x1), x);
        vs = fma(h, fma(a32, v2, a31 * v1), v);
        RHS(xs, vs, x3, v3);
        xs = fma(h, fma(a43, x3, a41 * x1), x);
        vs = fma(h, fma(a43, v3, a41 * v1), v);
        RHS(xs, vs, x4, v4);
        xs = fma(h, fma(a54, x4, fma(a53, x3, a51 * x1)), x);
        vs = fma(h, fma(a54, v4, fma(a53, v3, a51 * v1)), v);
        RHS(xs, vs, x5, v5);
        xs = fma(h, fma(a65, x5, fma(a64, x4, a61 * x1)), x);
        vs = fma(h, fma(a65, v5, fma(a64, v4, a61 * v1)), v);
        RHS(xs, vs, x6, v6);
        xs = fma(h, fma(a76, x6, fma(a75, x5, fma(a74, x4, a71 * x1))), x);
        vs = fma(h, fma(a76, v6, fma(a75, v5, fma(a74, v4, a71 * v1))), v);
        RHS(xs, vs, x7, v7);
        STAGE(fma(a87, k7, fma(a86, k6, fma(a85, k5, fma(a84, k4, a81 * k1)))));
        RHS(xs, vs, x8, v8);
        STAGE(fma(a98, k8, fma(a97, k7, fma(a96, k6, fma(a95, k5, fma(a94, k4, a91 * k1))))));
        RHS(xs, vs, x9, v9);
        STAGE(fma(a109, k9, fma(a108, k8, fma(a107, k7, fma(a106, k6, fma(a105, k5, fma(a104, k4, a101 * k1)))))));
        RHS(xs, vs, x10, v10);
        STAGE(fma(a1110, k10, fma(a119, k9, fma(a118, k8, fma(a117, k7, fma(a116, k6, fma(a115, k5, fma(a114, k4, a111 * k1))))))));
        RHS(xs, vs, x2, v2);
        const double tph = tx + h;
        STAGE(fma(a1211, k2, fma(a1210, k10, fma(a129, k9, fma(a128, k8, fma(a127, k7, fma(a126, k6, fma(a125, k5, fma(a124, k4,
                  a121 * k1)))))))));
        RHS(xs, vs, x3, v3);
        nfcn += 11;

        // the new state and the error estimates (:410-444)
        double err = 0.0, err2 = 0.0;
#define UPDATE(p, pn)                                                                                                  \
    do {                                                                                                               \
        GX_K(p)                                                                                                        \
        const double bs = fma(b12, k3, fma(b11, k2, fma(b10, k10, fma(b9, k9, fma(b8, k8, fma(b7, k7, fma(b6, k6,       \
                              b1 * k1)))))));                                                                          \
        pn = fma(h, bs, p);                                                                                            \
        const double isk = fast::rcp_f(fma(rtoli, max_abs(p, pn), atoli));                                             \
        double q = fma(-bhh3, k3, fma(-bhh2, k9, fma(-bhh1, k1, bs))) * isk;                                           \
        err2 = fma(q, q, err2);                                                                                        \
        q = fma(er12, k3, fma(er11, k2, fma(er10, k10, fma(er9, k9, fma(er8, k8, fma(er7, k7, fma(er6, k6,              \
                er1 * k1))))))) * isk;                                                                                 \
        err = fma(q, q, err);                                                                                          \
    } while (0)
        UPDATE(x, xn);
        UPDATE(v, vn);
#undef UPDATE
        if (!active) err = err2 = 0.0;
        axis_sum2(err, err2, buf[par], B);
        par ^= 1;
        double deno = fma(0.01, err2, err);
        if (deno <= 0.0) deno = 1.0;
        err = fabs(h) * err * dsqrt(ddiv(1.0, deno * nsys));
        // computation of hnew (:446-452); gala's pow(err, 1/8) (beta = 0) as three square roots
        const double fac11 = dsqrt(dsqrt(dsqrt(err)));
        const double fac = max_d(facc2, min_d(facc1, ddiv(fac11, safe)));
        double hnew = ddiv(h, fac);
        if (err <= 1.0) {
            naccpt++;
            double fx, fv;
            RHS(xn, vn, fx, fv);
            nfcn++;

            // stiffness detection (:463-486); like gala, the first detection returns -4
            const bool due = --to_test == 0;
            if (due) to_test = nstiff;
            if (due || (iasti > 0)) {
                double q = fx - x3, p = fv - v3;
                double stnum = active ? fma(q, q, p * p) : 0.;
                q = xn - xs;
                p = vn - vs;
                double stden = active ? fma(q, q, p * p) : 0.;
                axis_sum2(stnum, stden, buf[par], B);
                par ^= 1;
                if (stden > 0.0) hlamb = h * dsqrt(ddiv(stnum, stden));
                if (hlamb > 6.1) {
                    nonsti = 0;
                    iasti++;
                    idid = -4;
                    break;
                }
                nonsti++;
                if (nonsti == 6) iasti = 0;
            }

            // output times inside [xold, xold + hout] (see gx_dop853.cu)
            int64_t out_end = out_idx;
            if (A.save_all) {
                const double e0 = xold, e1 = e0 + hout;
                while (out_end < A.ntimes) {
                    const double t_out = t[out_end];
                    if (!((e0 <= t_out && t_out <= e1) || (e1 <= t_out && t_out <= e0))) break;
                    out_end++;
                }
            }
            if (A.save_all && kept < out_end) {
                // dense output preparation (:492-582)
#define D8(d, k4_)                                                                                                  \
    fma(d##12, k3, fma(d##11, k2, fma(d##10, k10, fma(d##9, k9, fma(d##8, k8, fma(d##7, k7, fma(d##6, k6, d##1 * k1)))))))
#define PREP(p, f)                                                                                                  \
    double p##r5, p##r6, p##r7, p##r8, p##s14;                                                                      \
    {                                                                                                               \
        GX_K(p)                                                                                                     \
        p##r5 = fma(d413, f, D8(d4, f));                                                                            \
        p##r6 = fma(d513, f, D8(d5, f));                                                                            \
        p##r7 = fma(d613, f, D8(d6, f));                                                                            \
        p##r8 = fma(d713, f, D8(d7, f));                                                                            \
        p##s14 = fma(h, fma(a1413, f, fma(a1412, k3, fma(a1411, k2, fma(a1410, k10, fma(a149, k9, fma(a148, k8,      \
                            fma(a147, k7, a141 * k1))))))), p);                                                     \
    }
                PREP(x, fx)
                PREP(v, fv)
                double x14, v14, x15, v15, x16, v16;
                RHS(xs14, vs14, x14, v14);
#define S15(p, f) \
    fma(h, fma(a1514, p##14, fma(a1513, f, fma(a1512, p##3, fma(a1511, p##2, fma(a158, p##8, fma(a157, p##7, fma(a156, p##6, \
        a151 * p##1))))))), p)
                RHS(S15(x, fx), S15(v, fv), x15, v15);
#define S16(p, f) \
    fma(h, fma(a1615, p##15, fma(a1614, p##14, fma(a1613, f, fma(a169, p##9, fma(a168, p##8, fma(a167, p##7, fma(a166, p##6, \
        a161 * p##1))))))), p)
                RHS(S16(x, fx), S16(v, fv), x16, v16);
                nfcn += 3;
#define FIN(p, f, pn)                                                                            \
    p##r5 = h * fma(d416, p##16, fma(d415, p##15, fma(d414, p##14, p##r5)));                     \
    p##r6 = h * fma(d516, p##16, fma(d515, p##15, fma(d514, p##14, p##r6)));                     \
    p##r7 = h * fma(d616, p##16, fma(d615, p##15, fma(d614, p##14, p##r7)));                     \
    p##r8 = h * fma(d716, p##16, fma(d715, p##15, fma(d714, p##14, p##r8)));                     \
    const double p##d = pn - p, p##b = fma(h, p##1, -p##d), p##r4 = fma(-h, f, p##d) - p##b;
                FIN(x, fx, xn)
                FIN(v, fv, vn)
#undef FIN
#undef S16
#undef S15
#undef PREP
#undef D8
                double *ox = out + (axis * A.n_out + out_slot) * n + i0 + j;
                double *ov = out + ((3 + axis) * A.n_out + out_slot) * n + i0 + j;
                for (; kept < out_end; kept += A.out_stride, out_slot++) {
                    const double s = ddiv(t[kept] - xold, hout);
                    const double s1 = 1.0 - s;
#define DENSE(p) \
    fma(s, fma(s1, fma(s, fma(s1, fma(s, fma(s1, fma(s, p##r8, p##r7), p##r6), p##r5), p##r4), p##b), p##d), p)
                    const double yx = DENSE(x), yv = DENSE(v);
#undef DENSE
                    if (active) {
                        __stcs(ox, yx);
                        __stcs(ov, yv);
                    }
                    ox += n;
                    ov += n;
                }
            }
            out_idx = out_end;

            x1 = fx;
            v1 = fv;
            x = xn;
            v = vn;
            tx = tph;
            if (last) {
                idid = 1;
                break;
            }
            if (fabs(hnew) > hmax) hnew = posneg * hmax;
            if (reject) hnew = posneg * min_d(fabs(hnew), fabs(h));
            reject = 0;
        } else {
            hnew = ddiv(h, min_d(facc1, ddiv(fac11, safe)));
            reject = 1;
            if (naccpt >= 1) nrejct = nrejct + 1;
            last = 0;
        }
        h = hnew;
    }
#undef STAGE
#undef GX_K
    if (B.T > 1) cluster_sync_all();  // no CTA leaves while another may still write to it

    if (!A.save_all && active) {
        out[axis * n + i0 + j] = x;
        out[(3 + axis) * n + i0 + j] = v;
    }
    if (B.wi == 0 && lane == 0) {
        status[b] = idid;
        if (stats) {
            stats[4 * b + 0] = nfcn;
            stats[4 * b + 1] = nstep;
            stats[4 * b + 2] = naccpt;
            stats[4 * b + 3] = nrejct;
        }
    }
}
#undef RHS

// Warps of a batch, eight orbits each.
static int axis_warps(const DopArgs &A, int64_t n) { return (int)(((A.nbatch < n ? A.nbatch : n) + 7) / 8); }

// Whether the potential's components go one to a lane.
static bool one_per_lane(const DevPot &dp) {
    bool lanes = dp.ncomp <= 4;
    for (int i = 0; i < dp.ncomp && lanes; i++) lanes = !dp.c[i].do_sr;
    return lanes;
}

bool dop853_axis_takes(const DevPot &dp, const DevFrame &df, const DopArgs &A, int64_t n) {
    if (dp.has_scf || dp.cdev) return false;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return false;
    const int64_t nbatches = (n + A.nbatch - 1) / A.nbatch;
    const int T = axis_warps(A, n);
    // Batches of at most 16 orbits share warps in the general kernel.  The lines lie
    // where the SMs' FP64 units are full: 400 steps of 0.5 Myr, batches of 100, one lane
    // per orbit / here, ms: static MW composite 1,000 orbits 14.4 / 8.8, 7,000
    // 14.4 / 12.8, 9,000 14.6 / 20.0; rotating bar 37 17.4 / 6.1, 1,000 39.3 / 10.6,
    // 9,000 44.2 / 24.8, 12,000 43.4 / 29.2 (components one to a lane; one after the
    // other 9,000 take 43.6).
    const int64_t most = (df.type != GX_FRAME_STATIC && one_per_lane(dp) ? 14 : 6) * (int64_t)sms;
    return T <= AXIS_MAX_WARPS && (A.nbatch > 16 || nbatches == 1) && nbatches * T <= most;
}

int launch_dop853_axis(const DevPot &dp, const DevFrame &df, const DopArgs &A, const double *w0, int64_t n, const double *t,
                       double *out, int32_t *status, int64_t *stats, cudaStream_t st) {
    const int T = axis_warps(A, n), W = T <= 8 ? 1 : T <= 16 ? 2 : 4, G = (T + W - 1) / W;
    const int64_t nbatches = (n + A.nbatch - 1) / A.nbatch;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(nbatches * G));
    cfg.blockDim = dim3(32 * W);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = G;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    const bool rot = df.type != GX_FRAME_STATIC;
    const auto kernel = one_per_lane(dp) ? (rot ? dop853_axis_kernel<true, true> : dop853_axis_kernel<true, false>)
                               : (rot ? dop853_axis_kernel<false, true> : dop853_axis_kernel<false, false>);
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, dp, df, A, G, w0, n, t, out, status, stats);
    if (e != cudaSuccess) {
        set_error("dop853 launch failed: %s", cudaGetErrorString(e));
        return GX_ERR_CUDA;
    }
    return check_launch("dop853");
}

}  // namespace gx
