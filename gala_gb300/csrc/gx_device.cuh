// gx_device.cuh -- device-side potential, frame and Hamiltonian evaluation.
//
// Every evaluation function is instantiated twice: SCF = false for potentials
// made only of closed-form components (all state stays in registers) and
// SCF = true when an SCF component is present (the SCF series is an
// out-of-line call, which forces the caller's small arrays into local memory).
//
// The potential is handed to every kernel BY VALUE (DevPot below, a few KB of
// kernel parameters that sit in the constant bank): component type tags,
// shift/rotate data and up to GX_MAX_INLINE_PARAMS packed parameters.  Large
// parameter blocks (SCF coefficients) stay in global memory behind `pdev`.
//
// Every FP64 expression below keeps gala's evaluation order (the cited
// *_gradient_single / *_value functions of
// src/gala/potential/potential/builtin/builtin_potentials.cpp); the FP64
// translation units are compiled with -fmad=false so that no multiply-add is
// contracted, which makes the results operation-for-operation those of gala's
// C code built without contraction.  The square roots and quotients come from
// the integer pipe (gx_ipipe.cuh: correctly rounded, so the same bits as the FP64
// instructions they replace, 8 FP64-pipe instructions each) and so does ln (within
// 0.65 ulp, the library's is within 1); products of parameters are formed once on
// the host, and the radius once per point for all components that are neither
// shifted nor rotated.  An MW-composite gradient takes 51 FP64-pipe instructions
// that way instead of about 200.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/gala_gb300.h"
#include "gx_ipipe.cuh"

namespace gx {

struct DevComp {
    int32_t type;
    int32_t do_sr;
    int32_t poff;     // offset of this component's [G, ...] in DevPot::p (inline) or pdev
    int32_t inl;      // 1: parameters are in DevPot::p; 0: in pdev (SCF)
    double q0[3];
    double R[9];
    // Constants derived from the parameters on the host, each the IEEE result of
    // gala's own expression where gala forms it: dc[0] = G m; Plummer,
    // Miyamoto-Nagai: dc[1] = b^2; NFW: dc[1] = 1 / r_s, dc[2..4] = 1 / a^2,
    // 1 / b^2, 1 / c^2 (1 where the shape has no such axis), dc[5] = G m / r_s,
    // dc[6] = r_s^2.
    double dc[7];
};

struct DevPot {
    int32_t ncomp;
    int32_t n_inline;
    int32_t has_scf;      // selects the SCF = true instantiation on the host
    int32_t regular;      // see finite_gradient below
    const double *pdev;   // device copy of the packed parameters (may be null)
    const DevComp *cdev;  // component table in device memory (more than
                          // GX_MAX_COMPONENTS components), else null
    int32_t dbh;          // a disk-bulge-halo composite: see d
    int32_t dbh_order;    // and its order: 1 spheres, disk, halo; 2 disk, spheres, halo; 0 another
    int32_t sphere;       // GX_POT_HERNQUIST for one unshifted Hernquist sphere (d.gm1, d.c1), else 0
    int32_t pad;
    DevComp c[GX_MAX_COMPONENTS];
    double p[GX_MAX_INLINE_PARAMS];
    // Constants of a disk-bulge-halo composite: one or two Hernquist spheres, one
    // Miyamoto-Nagai disk and one spherical NFW halo, in any order, none shifted or
    // rotated (a missing second sphere has mass 0).  fast::dbh_gradient evaluates
    // such a composite in one straight run.
    struct {
        double gm1, c1, gm2, c2;  // spheres
        double gmd, a, b2;        // disk
        double gmh, irs;          // halo: G m, 1 / r_s
        double vh2, rs, rs2;      // halo, as gala's expressions take it: G m / r_s, r_s, r_s^2
    } d;
};

// A large composite seen through its device table: the same members as DevPot
// (c, p, pdev, ncomp), so the component evaluators below serve both; every
// table component reads its parameters from the device copy (inl == 0).
struct TabPot {
    int32_t ncomp;
    const DevComp *c;
    const double *p;
    const double *pdev;
};

__device__ __forceinline__ TabPot table_view(const DevPot &pot) { return TabPot{pot.ncomp, pot.cdev, pot.pdev, pot.pdev}; }

struct DevFrame {
    int32_t type;   // gx_frame_type
    int32_t pad;
    double O[3];
};

// ---------------------------------------------------------------------------
// SCF (src/gala/potential/scf/src/bfe.cpp:114-259, bfe_helper.cpp:14-90).
// Implemented in gx_scf.cuh; declared here so the component switch can call it.
// ---------------------------------------------------------------------------
static __device__ double scf_value_dev(const double *p, const double *q);
static __device__ void scf_gradient_dev(const double *p, const double *q, double *g);
static __device__ double scf_density_dev(const double *p, const double *q);

__device__ __forceinline__ double norm3_sq(const double *q) {
    return q[0] * q[0] + q[1] * q[1] + q[2] * q[2];
}

// gala's sqrt(x), a / b and log(x).  LIBLN takes the library's ln instead of the
// integer one (30 FP64-pipe instructions more per NFW gradient; one evaluation in
// 300 differs in the last bit).  The Leapfrog n-body kernels ask for it, and so
// does every potential value: stream particles bound to a light progenitor move
// chaotically at Leapfrog's step, so a last-bit change of the force, or of the
// second difference of Phi that places them, moves a few of them by 1e-3 kpc.
__device__ __forceinline__ double dsqrt(double x) { return ip::sqrt_rn(x); }
__device__ __forceinline__ double ddiv(double a, double b) { return ip::div_rn(a, b); }
template <bool LIBLN>
__device__ __forceinline__ double dlog(double x) {
    if (!LIBLN && ip::ln_range(x)) return ip::ln_n(x);
    return log(x);
}

// Powers in the gradients.  gala calls pow(x, -1.5) (Miyamoto-Nagai) and
// pow(r, 3.0) (Kepler).  The FP64 pow of CUDA runs an extended-precision log
// and exp, a hundred-odd instructions on the FP64 pipe, whose rate on this part
// is 1/64 of FP32.  1 / (x sqrt(x)) is correctly rounded in each of its three
// operations (within 1.5 ulp of x^-1.5) and r r r within 1 ulp of r^3: the
// accuracy class of pow itself, which does not round like the host's pow
// either.  Edge values match pow: 0 -> inf, inf -> 0, NaN -> NaN.
__device__ __forceinline__ double pow_m1p5(double x) { return ddiv(1.0, x * dsqrt(x)); }
__device__ __forceinline__ double cube(double r) { return r * r * r; }

// x^2 + y^2 + z^2 and its root at one point, formed when a component first asks
// for them and kept for the others at the same point (the same expressions, so
// the same bits).
struct Radius {
    double s, r;
    int have;  // 1: s, 2: s and r
    __device__ __forceinline__ double sq(const double *q) {
        if (have == 0) {
            s = norm3_sq(q);
            have = 1;
        }
        return s;
    }
    __device__ __forceinline__ double root(const double *q) {
        if (have < 2) {
            r = dsqrt(sq(q));
            have = 2;
        }
        return r;
    }
};

// Whether the gradient at x is finite for certain, so that gala's product of it
// with a zero coefficient (the first sub-step of Ruth4) is zero: `regular` says
// that every component is a closed form centred on the origin with parameters of
// ordinary size (regular_component in gx_host.cu), and the largest coordinate
// lies within 2^-100 and 2^100.
__device__ __forceinline__ bool ordinary(double v) {
    return ((unsigned)__double2hiint(v) & 0x7fffffffu) - (923u << 20) < (200u << 20);
}
__device__ __forceinline__ bool finite_gradient(const DevPot &pot, const double *x) {
    const unsigned m = 0x7fffffffu;
    const unsigned h = max((unsigned)__double2hiint(x[0]) & m, max((unsigned)__double2hiint(x[1]) & m, (unsigned)__double2hiint(x[2]) & m));
    return pot.regular && h - (923u << 20) < (200u << 20);
}

// Parameters of component ci as a plain pointer: inline ones are read from the
// kernel-parameter copy, SCF blocks from global memory.
#define GX_PARAM(pot, ci, k) ((pot).c[ci].inl ? (pot).p[(pot).c[ci].poff + (k)] : (pot).pdev[(pot).c[ci].poff + (k)])

// Value of one component at q (kepler_value :58-64, hernquist_value :211-219,
// plummer_value :292-300, miyamotonagai_value :1287-1296, sphericalnfw_value
// :819-833, flattenednfw_value :925-942, triaxialnfw_value :1028-1049).
template <bool SCF, typename PV>
__device__ __forceinline__ double comp_value(const PV &pot, int ci, const double *q, Radius &R) {
    const DevComp &C = pot.c[ci];
#define P(k) GX_PARAM(pot, ci, k)
    double u;
    switch (C.type) {
    case GX_POT_NULL:
        return 0.;
    case GX_POT_KEPLER:
        return ddiv(-C.dc[0], R.root(q));
    case GX_POT_HERNQUIST:
        return ddiv(-C.dc[0], R.root(q) + P(2));
    case GX_POT_PLUMMER:
        return ddiv(-C.dc[0], dsqrt(R.sq(q) + C.dc[1]));
    case GX_POT_MIYAMOTONAGAI: {
        const double zd = (P(2) + dsqrt(q[2] * q[2] + C.dc[1]));
        return ddiv(-C.dc[0], dsqrt(q[0] * q[0] + q[1] * q[1] + zd * zd));
    }
    case GX_POT_SPHERICALNFW:
        u = ddiv(R.root(q), P(2));
        break;
    case GX_POT_FLATTENEDNFW:
        u = ddiv(dsqrt(q[0] * q[0] + q[1] * q[1] + ddiv(q[2] * q[2], P(5) * P(5))), P(2));
        break;
    case GX_POT_TRIAXIALNFW:
        u = ddiv(dsqrt(ddiv(q[0] * q[0], P(3) * P(3)) + ddiv(q[1] * q[1], P(4) * P(4)) + ddiv(q[2] * q[2], P(5) * P(5))), P(2));
        break;
    case GX_POT_SCF:
        if constexpr (SCF) return scf_value_dev(pot.pdev + C.poff, q);
        return __longlong_as_double(0x7ff8000000000000LL);
    default:
        return __longlong_as_double(0x7ff8000000000000LL);
    }
    // the three NFW shapes (v_h^2 = -G m / r_s)
    if (u == 0) return -C.dc[5];
    return ddiv(-C.dc[5] * log(1 + u), u);
#undef P
}

// Gradient of one component, accumulated into g (kepler :66-76, hernquist
// :221-233, plummer :302-314, miyamotonagai :1298-1312, sphericalnfw :835-850,
// flattenednfw :944-962, triaxialnfw :1051-1072).
template <bool SCF, bool LIBLN, typename PV>
__device__ __forceinline__ void comp_gradient(const PV &pot, int ci, const double *q, double *g, Radius &R) {
    const DevComp &C = pot.c[ci];
#define P(k) GX_PARAM(pot, ci, k)
    double fac, u;
    switch (C.type) {
    case GX_POT_NULL:
        return;
    case GX_POT_KEPLER:
        fac = ddiv(C.dc[0], cube(R.root(q)));
        break;
    case GX_POT_HERNQUIST: {
        const double r = R.root(q);
        fac = ddiv(C.dc[0], (r + P(2)) * (r + P(2)) * r);
        break;
    }
    case GX_POT_PLUMMER: {
        const double R2b = R.sq(q) + C.dc[1];
        fac = ddiv(ddiv(C.dc[0], dsqrt(R2b)), R2b);
        break;
    }
    case GX_POT_MIYAMOTONAGAI: {
        const double sqrtz = dsqrt(q[2] * q[2] + C.dc[1]);
        const double zd = P(2) + sqrtz;
        fac = C.dc[0] * pow_m1p5(q[0] * q[0] + q[1] * q[1] + zd * zd);
        g[0] = g[0] + fac * q[0];
        g[1] = g[1] + fac * q[1];
        g[2] = g[2] + fac * q[2] * (1. + ddiv(P(2), sqrtz));
        return;
    }
    case GX_POT_SPHERICALNFW:
    case GX_POT_FLATTENEDNFW:
    case GX_POT_TRIAXIALNFW: {
        double m;
        if (C.type == GX_POT_SPHERICALNFW)
            m = R.root(q);
        else if (C.type == GX_POT_FLATTENEDNFW)
            m = dsqrt(q[0] * q[0] + q[1] * q[1] + ddiv(q[2] * q[2], P(5) * P(5)));
        else
            m = dsqrt(ddiv(q[0] * q[0], P(3) * P(3)) + ddiv(q[1] * q[1], P(4) * P(4)) + ddiv(q[2] * q[2], P(5) * P(5)));
        u = ddiv(m, P(2));
        const double u1 = 1 + u;
        fac = ddiv(ddiv(C.dc[5], u * u * u), C.dc[6]) * (dlog<LIBLN>(u1) - ddiv(u, u1));
        if (C.type == GX_POT_SPHERICALNFW) break;
        if (C.type == GX_POT_FLATTENEDNFW) {
            g[0] = g[0] + fac * q[0];
            g[1] = g[1] + fac * q[1];
        } else {
            g[0] = g[0] + ddiv(fac * q[0], P(3) * P(3));
            g[1] = g[1] + ddiv(fac * q[1], P(4) * P(4));
        }
        g[2] = g[2] + ddiv(fac * q[2], P(5) * P(5));
        return;
    }
    case GX_POT_SCF:
        if constexpr (SCF) {
            scf_gradient_dev(pot.pdev + C.poff, q, g);
            return;
        }
        fac = __longlong_as_double(0x7ff8000000000000LL);
        break;
    default: {
        const double nan = __longlong_as_double(0x7ff8000000000000LL);
        g[0] = nan; g[1] = nan; g[2] = nan;
        return;
    }
    }
    g[0] = g[0] + fac * q[0];
    g[1] = g[1] + fac * q[1];
    g[2] = g[2] + fac * q[2];
#undef P
}

// comp_gradient for one axis: the component `axis` of the gradient is increased in
// g, with q the coordinate and s0, s1, s2 the squares of all three (the same
// expressions as above, so the same bits).
template <typename PV>
__device__ __forceinline__ void comp_gradient_axis(const PV &pot, int ci, double s0, double s1, double s2, double q, int axis,
                                                   double &g, Radius &R) {
    const DevComp &C = pot.c[ci];
#define P(k) GX_PARAM(pot, ci, k)
    double fac;
    R.s = s0 + s1 + s2;
    if (R.have == 0) R.have = 1;
    const double *none = nullptr;
    switch (C.type) {
    case GX_POT_NULL:
        return;
    case GX_POT_KEPLER:
        fac = ddiv(C.dc[0], cube(R.root(none)));
        break;
    case GX_POT_HERNQUIST: {
        const double r = R.root(none);
        fac = ddiv(C.dc[0], (r + P(2)) * (r + P(2)) * r);
        break;
    }
    case GX_POT_PLUMMER: {
        const double R2b = R.s + C.dc[1];
        fac = ddiv(ddiv(C.dc[0], dsqrt(R2b)), R2b);
        break;
    }
    case GX_POT_MIYAMOTONAGAI: {
        const double sqrtz = dsqrt(s2 + C.dc[1]);
        const double zd = P(2) + sqrtz;
        fac = C.dc[0] * pow_m1p5(s0 + s1 + zd * zd);
        if (axis == 2)
            g = g + fac * q * (1. + ddiv(P(2), sqrtz));
        else
            g = g + fac * q;
        return;
    }
    case GX_POT_SPHERICALNFW:
    case GX_POT_FLATTENEDNFW:
    case GX_POT_TRIAXIALNFW: {
        double m;
        if (C.type == GX_POT_SPHERICALNFW)
            m = R.root(none);
        else if (C.type == GX_POT_FLATTENEDNFW)
            m = dsqrt(s0 + s1 + ddiv(s2, P(5) * P(5)));
        else
            m = dsqrt(ddiv(s0, P(3) * P(3)) + ddiv(s1, P(4) * P(4)) + ddiv(s2, P(5) * P(5)));
        const double u = ddiv(m, P(2)), u1 = 1 + u;
        fac = ddiv(ddiv(C.dc[5], u * u * u), C.dc[6]) * (dlog<false>(u1) - ddiv(u, u1));
        if (C.type == GX_POT_TRIAXIALNFW || (C.type == GX_POT_FLATTENEDNFW && axis == 2)) {
            const double a = P(3 + axis);
            g = g + ddiv(fac * q, a * a);
            return;
        }
        break;
    }
    default:
        g = __longlong_as_double(0x7ff8000000000000LL);
        return;
    }
    g = g + fac * q;
#undef P
}

// Density of one component (kepler_density :78-88, hernquist_density :235-244,
// plummer_density :316-324, miyamotonagai_density :1314-1332,
// sphericalnfw_density :852-864).  Flattened/triaxial NFW have no density in
// gala (nan_density).
template <bool SCF, typename PV>
__device__ __forceinline__ double comp_density(const PV &pot, int ci, const double *q) {
    const int type = pot.c[ci].type;
    const double PI = 3.14159265358979323846;
#define P(k) GX_PARAM(pot, ci, k)
    switch (type) {
    case GX_POT_NULL:
        return 0.;
    case GX_POT_KEPLER:
        return (norm3_sq(q) == 0.) ? __longlong_as_double(0x7ff0000000000000LL) : 0.;
    case GX_POT_HERNQUIST: {
        const double r = sqrt(norm3_sq(q));
        const double rho0 = P(1) / (2 * PI * P(2) * P(2) * P(2));
        return rho0 / ((r / P(2)) * pow(1 + r / P(2), 3.0));
    }
    case GX_POT_PLUMMER: {
        const double r2 = norm3_sq(q);
        return 3 * P(1) / (4 * PI * P(2) * P(2) * P(2)) * pow(1 + r2 / (P(2) * P(2)), -2.5);
    }
    case GX_POT_MIYAMOTONAGAI: {
        const double M = P(1), a = P(2), b = P(3);
        const double R2 = q[0] * q[0] + q[1] * q[1];
        const double sqrt_zb = sqrt(q[2] * q[2] + b * b);
        const double numer = (b * b * M / (4 * PI)) * (a * R2 + (a + 3 * sqrt_zb) * (a + sqrt_zb) * (a + sqrt_zb));
        const double denom = pow(R2 + (a + sqrt_zb) * (a + sqrt_zb), 2.5) * sqrt_zb * sqrt_zb * sqrt_zb;
        return numer / denom;
    }
    case GX_POT_SPHERICALNFW: {
        const double v_h2 = P(0) * P(1) / P(2);
        const double r = sqrt(norm3_sq(q));
        const double rho0 = v_h2 / (4 * PI * P(0) * P(2) * P(2));
        return rho0 / ((r / P(2)) * pow(1 + r / P(2), 2.0));
    }
    case GX_POT_SCF:
        if constexpr (SCF) return scf_density_dev(pot.pdev + pot.c[ci].poff, q);
        return __longlong_as_double(0x7ff8000000000000LL);
    default:
        return __longlong_as_double(0x7ff8000000000000LL);
    }
#undef P
}

// q' = R (q - q0) (apply_shift_rotate_N, cpotential.cpp:152-167).
__device__ __forceinline__ void shift_rotate(const DevComp &c, const double *q, double *qt) {
    const double x = q[0] - c.q0[0], y = q[1] - c.q0[1], z = q[2] - c.q0[2];
    qt[0] = c.R[0] * x + c.R[1] * y + c.R[2] * z;
    qt[1] = c.R[3] * x + c.R[4] * y + c.R[5] * z;
    qt[2] = c.R[6] * x + c.R[7] * y + c.R[8] * z;
}

// c_potential (cpotential.cpp:170-189).  The shifted path of gala builds q'
// as 0 + R0 x + ...; for finite values that equals R0 x + ..., bit for bit.
template <bool SCF, typename PV>
__device__ __forceinline__ double potential_value_t(const PV &pot, const double *q) {
    double v = 0;
    Radius R;
    R.have = 0;
    for (int i = 0; i < pot.ncomp; i++) {
        if (pot.c[i].do_sr == 0) {
            v = v + comp_value<SCF>(pot, i, q, R);
        } else {
            double qt[3];
            Radius Rt;
            Rt.have = 0;
            shift_rotate(pot.c[i], q, qt);
            v = v + comp_value<SCF>(pot, i, qt, Rt);
        }
    }
    return v;
}

// c_density (cpotential.cpp:192-211).
template <bool SCF, typename PV>
__device__ __forceinline__ double potential_density_t(const PV &pot, const double *q) {
    double v = 0;
    for (int i = 0; i < pot.ncomp; i++) {
        if (pot.c[i].do_sr == 0) {
            v = v + comp_density<SCF>(pot, i, q);
        } else {
            double qt[3];
            shift_rotate(pot.c[i], q, qt);
            v = v + comp_density<SCF>(pot, i, qt);
        }
    }
    return v;
}

// c_gradient at one point (cpotential.cpp:214-287): zero, accumulate each
// component in order; shifted/rotated components go through a zeroed
// temporary, are rotated back with R^T (apply_rotate_T, :103-134) and added.
template <bool SCF, bool LIBLN, typename PV>
__device__ __forceinline__ void potential_gradient_t(const PV &pot, const double *q, double *g) {
    g[0] = 0.; g[1] = 0.; g[2] = 0.;
    Radius R;
    R.have = 0;
    for (int i = 0; i < pot.ncomp; i++) {
        if (pot.c[i].do_sr == 0) {
            comp_gradient<SCF, LIBLN>(pot, i, q, g, R);
        } else {
            const DevComp &c = pot.c[i];
            double qt[3], gt[3] = {0., 0., 0.};
            Radius Rt;
            Rt.have = 0;
            shift_rotate(c, q, qt);
            comp_gradient<SCF, LIBLN>(pot, i, qt, gt, Rt);
            g[0] += c.R[0] * gt[0] + c.R[3] * gt[1] + c.R[6] * gt[2];
            g[1] += c.R[1] * gt[0] + c.R[4] * gt[1] + c.R[7] * gt[2];
            g[2] += c.R[2] * gt[0] + c.R[5] * gt[1] + c.R[8] * gt[2];
        }
    }
}

// The factors of a disk-bulge-halo composite's gradient in gala's expressions, in
// one straight run (see fast::dbh_gradient): spheres f1, f2, disk fd with mz on
// its z component, halo fn; s0, s1, s2 are the squares of the coordinates.  False
// where an argument is outside the integer forms' range (the second sphere's G m is
// +0 or inside it: pack_dbh in gx_host.cu).  The bits are those of comp_gradient; side
// by side the chains take 16,384 uneven FP64 orbits from 35.5 to 22.0 ms.
template <bool LIBLN>
__device__ __forceinline__ bool dbh_factors(const DevPot &pot, double s0, double s1, double s2, double &f1, double &f2,
                                            double &fd, double &mz, double &fn) {
    const double xy2 = s0 + s1;
    const double r2 = xy2 + s2, w = s2 + pot.d.b2;
    const double r = ip::sqrt_rn_u(r2), sz = ip::sqrt_rn_u(w);
    const double d1 = (r + pot.d.c1) * (r + pot.d.c1) * r, d2 = (r + pot.d.c2) * (r + pot.d.c2) * r;
    const double u = ip::div_rn_u(r, pot.d.rs);
    const double zd = pot.d.a + sz;
    const double W = xy2 + zd * zd;
    const double sW = ip::sqrt_rn_u(W), W3 = W * sW;
    const double u1 = 1 + u, u3 = u * u * u;
    const bool ok = ip::ok_sqrt(r2) & ip::ok_sqrt(w) & ip::ok_sqrt(W) & ip::ok_div(pot.d.gm1, d1) & ip::ok_rcp(d2) &
                    ip::ok_div(r, pot.d.rs) & ip::ok_rcp(W3) & ip::ok_div(pot.d.a, sz) & ip::ln_range(u1) & ip::ok_rcp(u1) &
                    ip::ok_div(pot.d.vh2, u3) & ip::ok_rcp(pot.d.rs2);
    f1 = ip::div_rn_u(pot.d.gm1, d1);
    f2 = __double_as_longlong(pot.d.gm2) == 0 ? 0. : ip::div_rn_u(pot.d.gm2, d2);
    fd = pot.d.gmd * ip::div_rn_u(1.0, W3);
    mz = 1. + ip::div_rn_u(pot.d.a, sz);
    const double L = LIBLN ? log(u1) : ip::ln_n(u1);
    const double v = ip::div_rn_u(pot.d.vh2, u3);
    fn = ip::div_rn_u(v, pot.d.rs2) * (L - ip::div_rn_u(u, u1));
    return ok & ip::ok_rcp(v);
}

// One component of the gradient of such a composite from its factors, summed in
// the composite's order.
__device__ __forceinline__ double dbh_sum(int order, double q, double f1, double f2, double fd, double mz, double fn) {
    const double gd = fd * q * mz;
    const double a = order == 1 ? 0. + f1 * q : 0. + gd;
    const double b = order == 1 ? a + f2 * q : a + f1 * q;
    const double c = order == 1 ? b + gd : b + f2 * q;
    return c + fn * q;
}

// The descriptor's components: the by-value array, or the device table of a
// large composite (the branch is uniform over the grid).
template <bool SCF>
__device__ __forceinline__ double potential_value(const DevPot &pot, const double *q) {
    if (pot.cdev) return potential_value_t<SCF>(table_view(pot), q);
    return potential_value_t<SCF>(pot, q);
}
template <bool SCF>
__device__ __forceinline__ double potential_density(const DevPot &pot, const double *q) {
    if (pot.cdev) return potential_density_t<SCF>(table_view(pot), q);
    return potential_density_t<SCF>(pot, q);
}
template <bool SCF, bool LIBLN = false>
__device__ __forceinline__ void potential_gradient(const DevPot &pot, const double *q, double *g) {
    if (pot.cdev) {
        potential_gradient_t<SCF, LIBLN>(table_view(pot), q, g);
        return;
    }
    if constexpr (!SCF) {
        if (pot.dbh_order) {
            double f1, f2, fd, mz, fn;
            if (dbh_factors<LIBLN>(pot, q[0] * q[0], q[1] * q[1], q[2] * q[2], f1, f2, fd, mz, fn)) {
                g[0] = dbh_sum(pot.dbh_order, q[0], f1, f2, fd, 1., fn);
                g[1] = dbh_sum(pot.dbh_order, q[1], f1, f2, fd, 1., fn);
                g[2] = dbh_sum(pot.dbh_order, q[2], f1, f2, fd, mz, fn);
                return;
            }
        }
    }
    potential_gradient_t<SCF, LIBLN>(pot, q, g);
}

// Frame energy: static_frame_hamiltonian (builtin_frames.cpp:8-16) or
// constant_rotating_frame_3d_hamiltonian (:78-94).
__device__ __forceinline__ double frame_energy(const DevFrame &fr, const double *w) {
    if (fr.type == GX_FRAME_STATIC) {
        double E = 0.;
        for (int i = 0; i < 3; i++) E += w[i + 3] * w[i + 3];
        return 0.5 * E;
    }
    double E = 0.;
    for (int i = 0; i < 3; i++) E += 0.5 * w[i + 3] * w[i + 3];
    const double Lx = w[1] * w[5] - w[2] * w[4];
    const double Ly = -w[0] * w[5] + w[2] * w[3];
    const double Lz = w[0] * w[4] - w[1] * w[3];
    return E - (fr.O[0] * Lx + fr.O[1] * Ly + fr.O[2] * Lz);
}

// Hamilton's equations at one point, Fwrapper_T -> hamiltonian_gradient_T
// (chamiltonian.cpp:38-57) with the frame gradient of builtin_frames.cpp:18-24
// (static) or :96-112 (rotating); the momentum half is multiplied by -1.
template <bool SCF>
__device__ __forceinline__ void hamiltonian_rhs(const DevPot &pot, const DevFrame &fr, const double *w, double *f) {
    double g[3];
    potential_gradient<SCF>(pot, w, g);
    if (fr.type == GX_FRAME_STATIC) {
        f[0] = w[3];
        f[1] = w[4];
        f[2] = w[5];
        f[3] = g[0] * -1;
        f[4] = g[1] * -1;
        f[5] = g[2] * -1;
    } else {
        const double *O = fr.O;
        double Cx = O[1] * w[2] - O[2] * w[1];
        double Cy = -O[0] * w[2] + O[2] * w[0];
        double Cz = O[0] * w[1] - O[1] * w[0];
        f[0] = 0. + w[3] - Cx;
        f[1] = 0. + w[4] - Cy;
        f[2] = 0. + w[5] - Cz;
        Cx = O[1] * w[5] - O[2] * w[4];
        Cy = -O[0] * w[5] + O[2] * w[3];
        Cz = O[0] * w[4] - O[1] * w[3];
        f[3] = (g[0] + Cx) * -1;
        f[4] = (g[1] + Cy) * -1;
        f[5] = (g[2] + Cz) * -1;
    }
}

// Out-of-line entry points for the integrator kernels.  A kernel calls the
// potential many times per step (up to 16 for DOP853); calling one compiled
// copy instead of inlining every call keeps code size and compile time small.
// Arguments and results are passed by value so they stay in registers.
struct V3 {
    double v[3];
};
struct V6 {
    double v[6];
};

template <bool SCF, bool LIBLN = false>
__device__ __noinline__ V3 gradient_call(const DevPot &pot, V3 q) {
    V3 g;
    potential_gradient<SCF, LIBLN>(pot, q.v, g.v);
    return g;
}

// Lane k's value in each group of four lanes.
__device__ __forceinline__ double quad(double v, int k) { return __shfl_sync(0xffffffffu, v, k, 4); }

// The gradient's component `axis` at a point held by four lanes of a warp (lane c of
// the group holds coordinate min(c, 2); axis is the lane's).  Closed-form components
// in the by-value descriptor only.  All 32 lanes of the warp take part: with a mask
// per group every shuffle would wait on a synchronisation of its own.
static __device__ __noinline__ double gradient_axis_call(const DevPot &pot, double q, int axis) {
    const double s = q * q;
    const double s0 = quad(s, 0), s1 = quad(s, 1), s2 = quad(s, 2);
    double g = 0.;
    Radius R;
    R.have = 0;
    for (int i = 0; i < pot.ncomp; i++) {
        if (pot.c[i].do_sr == 0) {
            comp_gradient_axis(pot, i, s0, s1, s2, q, axis, g, R);
        } else {
            const DevComp &c = pot.c[i];
            double qf[3], qt[3], gt[3] = {0., 0., 0.};
            for (int k = 0; k < 3; k++) qf[k] = quad(q, k);
            Radius Rt;
            Rt.have = 0;
            shift_rotate(c, qf, qt);
            comp_gradient<false, false>(pot, i, qt, gt, Rt);
            g += c.R[axis] * gt[0] + c.R[3 + axis] * gt[1] + c.R[6 + axis] * gt[2];
        }
    }
    return g;
}

// Straight runs of the same for the composites that have one: MODE 1 a Hernquist
// sphere, 2 and 3 a disk-bulge-halo composite (dbh_order 1 and 2); 0 the general
// form.  Constants that differ by lane are read once per launch (AxisLane), and
// choices between lanes are selections: a branch would end the run in which the
// integer chains overlap.
struct AxisLane {
    double cc, num;  // the lane's sphere radius and numerator
    bool first, sphere, halo, z;
};
__device__ __forceinline__ double pick(bool p, double a, double b) {
    return __hiloint2double(p ? __double2hiint(a) : __double2hiint(b), p ? __double2loint(a) : __double2loint(b));
}
__device__ __forceinline__ AxisLane axis_lane(const DevPot &pot) {
    const int c = threadIdx.x & 3;
    AxisLane L;
    L.cc = c == 0 ? pot.d.c1 : pot.d.c2;
    // a missing second sphere: 1 / d, taken as 0 below
    L.num = c == 0 ? pot.d.gm1 : c == 1 ? (pot.d.gm2 == 0. ? 1. : pot.d.gm2) : pot.d.a;
    L.first = c == 0;
    L.sphere = c < 2;
    L.halo = c == 2;
    L.z = c >= 2;
    return L;
}

// False, for the whole warp, where an argument of a lane that counts is outside the
// integer forms' range: the caller goes on with the general form (a call here would
// make every value alive around it spill).
template <int MODE>
__device__ __forceinline__ bool gradient_axis(const DevPot &pot, const AxisLane &A, bool counts, double q, double &g) {
    const double s = q * q;
    const double s0 = quad(s, 0), s1 = quad(s, 1), s2 = quad(s, 2);
    bool ok;
    if constexpr (MODE == 1) {
        const double r2 = s0 + s1 + s2;
        const double r = ip::sqrt_rn_u(r2);
        const double d = (r + pot.d.c1) * (r + pot.d.c1) * r;
        ok = ip::ok_sqrt(r2) & ip::ok_div(pot.d.gm1, d);
        g = 0. + ip::div_rn_u(pot.d.gm1, d) * q;
    } else {
        // dbh_factors with the integer work shared out: of two square roots, and of
        // four and three quotients, each lane forms one
        const double xy2 = s0 + s1;
        const double a1 = pick(A.first || A.halo, xy2 + s2, s2 + pot.d.b2);
        const double q1 = ip::sqrt_rn_u(a1);
        const double r = quad(q1, 0), sz = quad(q1, 1);
        const double rc = r + A.cc;
        const double num = pick(A.halo, r, A.num), den = pick(A.sphere, rc * rc * r, pick(A.halo, pot.d.rs, sz));
        const double zd = pot.d.a + sz;
        const double W = xy2 + zd * zd;
        const double q2 = ip::div_rn_u(num, den);
        const double W3 = W * ip::sqrt_rn_u(W);
        const double f1 = quad(q2, 0), f2s = quad(q2, 1);
        const double u = quad(q2, 2), mz = 1. + quad(q2, 3);
        const double f2 = pick(__double_as_longlong(pot.d.gm2) == 0, 0., f2s);
        const double u1 = 1 + u, u3 = u * u * u;
        const double num3 = pick(A.z, u, pick(A.first, 1.0, pot.d.vh2));
        const double den3 = pick(A.z, u1, pick(A.first, W3, u3));
        const double q3 = ip::div_rn_u(num3, den3);
        const double L = ip::ln_n(u1);
        const double v = quad(q3, 1);
        const double fd = pot.d.gmd * quad(q3, 0);
        const double fn = ip::div_rn_u(v, pot.d.rs2) * (L - quad(q3, 2));
        ok = ip::ok_sqrt(a1) & ip::ok_div(num, den) & ip::ok_sqrt(W) & ip::ok_div(num3, den3) & ip::ln_range(u1) &
             ip::ok_div(v, pot.d.rs2);
        const double gd = fd * q * pick(A.z, mz, 1.0);
        g = MODE == 2 ? 0. + f1 * q + f2 * q + gd + fn * q : 0. + gd + f1 * q + f2 * q + fn * q;
    }
    return __all_sync(0xffffffffu, ok | !counts);
}

template <bool SCF>
__device__ __noinline__ V6 rhs_call(const DevPot &pot, const DevFrame &fr, V6 w) {
    V6 f;
    hamiltonian_rhs<SCF>(pot, fr, w.v, f.v);
    return f;
}

}  // namespace gx
