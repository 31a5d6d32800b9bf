// gx_fast64.cuh -- the FP64 force in instructions the FP64 pipe can afford.
//
// The FP64 unit takes one warp instruction per 19 cycles of an SM (76 of a
// sub-partition), and the library forms of the special operations are long
// sequences on it: sqrt and a/b cost 8 FP64-pipe instructions each, 1/x 5,
// log ~30, pow ~84 (measured with ncu instruction counters).  The adaptive
// DOP853 kernels, which evaluate the force 12 to 16 times a step and cannot be
// bit-identical to gala anyway (their step control runs pow), use the forms
// below instead of gala's literal expressions:
//
//   * sqrt, 1/x and ln run on the integer pipe (gx_ipipe.cuh): none of them
//     costs an FP64-pipe instruction in its usual range.  With FP32-seeded Newton
//     forms (5, 4 and 14 FP64 instructions) an MW composite right-hand side took
//     106 of them, with these 47 (DOP853 of 20,011 MW orbits x 1 Gyr: 232.9 ->
//     180.3 ms), and 33 with one radius and one factor for all its components
//     (Diag below);
//   * every a/b becomes a * (1/b) and products and sums are fused (fma);
//   * gala's formulas are rearranged algebraically where that removes an
//     operation (the NFW factor v_h^2 / u^3 / r_s^2 is G m / r^3, etc.).
// The results differ from gala's expressions by a few ulp per evaluation; the
// integrated orbits are checked against the oracle at 1e-12 relative.
#pragma once

#include "gx_device.cuh"
#include "gx_ipipe.cuh"
#include "gx_log_table.cuh"

namespace gx {
namespace fast {

// sqrt(u) and 1/x within 0.51 ulp, on the integer pipe.
__device__ __forceinline__ double sqrt_f(double u) { return ip::sqrt_n(u); }
__device__ __forceinline__ double rcp_f(double x) { return ip::rcp_n(x); }

// ln x, Tang's table-driven method (P. T. P. Tang, ACM TOMS 16, 1990): x = 2^k m
// with m in [1, 2), c_j = 1 + j/64 the nearest table point (j = 0..64), f = m - c_j
// (exact), r = f / c_j as f * (1 / c_j), and ln x = k ln 2 + ln c_j + ln(1 + r)
// with |r| <= 1/128 and ln(1 + r) from its Taylor series through r^9 (truncation
// below 2^-60 relative).  ln c_j and ln 2 come in high and low parts
// (gx_log_table.cuh, from 60-digit arithmetic).  About an ulp; 14 FP64-pipe
// instructions against ~30 for the library log.  It serves arguments below
// 1 + 2^-6, where the integer form's fixed-point sum would lose relative
// accuracy; zero, negative, subnormal, infinite and NaN arguments go to the
// library.
__device__ __forceinline__ double log_f(double x) {
    if (ip::ln_range(x)) return ip::ln_n(x);
    const int hi = __double2hiint(x), lo = __double2loint(x);
    if (hi < 0x00100000 || hi >= 0x7ff00000) return log(x);
    const int k = (hi >> 20) - 1023;
    const int mant = hi & 0x000fffff;
    const int j = (mant + (1 << 13)) >> 14;  // nearest multiple of 1/64
    const double m = __hiloint2double(0x3ff00000 | mant, lo);
    const double c = __hiloint2double(0x3ff00000 + (j << 14), 0);
    const double r = (m - c) * __ldg(&LOG_TAB[j][0]);
    // ln(1 + r) = r (1 - r/2 + r^2/3 - ... + r^8/9)
    double p = 1.0 / 9;
    p = fma(p, r, -1.0 / 8);
    p = fma(p, r, 1.0 / 7);
    p = fma(p, r, -1.0 / 6);
    p = fma(p, r, 1.0 / 5);
    p = fma(p, r, -1.0 / 4);
    p = fma(p, r, 1.0 / 3);
    p = fma(p, r, -0.5);
    const double l1r = fma(p * r, r, r);
    // k as a double from its bits (2^52 + 2^31 + k, minus the offset)
    const double kd = __hiloint2double(0x43300000, (int)(0x80000000u ^ (unsigned)k)) - 4503601774854144.0;
    const double lo_part = fma(kd, LN2_LO, __ldg(&LOG_TAB[j][2]) + l1r);
    return fma(kd, LN2_HI, __ldg(&LOG_TAB[j][1])) + lo_part;
}

// What one evaluation point's components share and add to: the radius (formed when
// a component first asks for it) and the diagonal factors of the gradient,
// g = ((F + A0) x, (F + A1) y, (F + A2) z).
struct Diag {
    double xy2, r2, r, ir;  // x^2 + y^2, its sum with z^2, the root and its reciprocal
    double F, A[3];
    bool have, aniso;
    __device__ __forceinline__ void init(const double *q) {
        xy2 = fma(q[0], q[0], q[1] * q[1]);
        r2 = fma(q[2], q[2], xy2);
        F = A[0] = A[1] = A[2] = 0.;
        have = aniso = false;
    }
    __device__ __forceinline__ void radius() {
        if (!have) r = ip::sqrt_rsqrt_n(r2, ir);
        have = true;
    }
    __device__ __forceinline__ void gradient(const double *q, double *g) const {
        if (aniso) {
            g[0] = (F + A[0]) * q[0];
            g[1] = (F + A[1]) * q[1];
        } else {
            g[0] = F * q[0];
            g[1] = F * q[1];
        }
        g[2] = (F + A[2]) * q[2];
    }
};

// Gradient of one closed-form component, added to the diagonal factors; the same
// cases and gala references as comp_gradient in gx_device.cuh.  Every one of them
// is a factor times the position, so a spherical component costs 4 to 7 FP64
// instructions instead of the 13 to 17 it took with a radius, a reciprocal and
// three accumulations of its own: an MW composite 33 instead of 47.
template <typename PV>
__device__ __forceinline__ void comp_gradient_f(const PV &pot, int ci, const double *q, Diag &d) {
    const DevComp &C = pot.c[ci];
    const int type = C.type;
#define P(k) GX_PARAM(pot, ci, k)
    switch (type) {
    case GX_POT_NULL:
        return;
    case GX_POT_KEPLER:
        d.radius();
        d.F = fma(C.dc[0] * d.ir, d.ir * d.ir, d.F);
        return;
    case GX_POT_HERNQUIST: {
        d.radius();
        const double rc = d.r + P(2);
        d.F = fma(C.dc[0], rcp_f(rc * rc * d.r), d.F);
        return;
    }
    case GX_POT_PLUMMER: {
        double i;
        ip::sqrt_rsqrt_n(d.r2 + C.dc[1], i);
        d.F = fma(C.dc[0] * i, i * i, d.F);
        return;
    }
    case GX_POT_MIYAMOTONAGAI: {
        double isz, i;
        const double sqrtz = ip::sqrt_rsqrt_n(fma(q[2], q[2], C.dc[1]), isz);
        const double zd = P(2) + sqrtz;
        ip::sqrt_rsqrt_n(fma(zd, zd, d.xy2), i);
        const double f = C.dc[0] * i * (i * i);
        d.F += f;
        d.A[2] = fma(f, P(2) * isz, d.A[2]);
        return;
    }
    case GX_POT_SPHERICALNFW:
    case GX_POT_FLATTENEDNFW:
    case GX_POT_TRIAXIALNFW: {
        // gala: v_h^2 / u^3 / r_s^2 (log(1 + u) - u / (1 + u)) with v_h^2 = G m / r_s
        // and u = m_r / r_s, m_r the (scaled) radius: G m / m_r^3 (...)
        double mr, im;
        if (type == GX_POT_SPHERICALNFW) {
            d.radius();
            mr = d.r;
            im = d.ir;
        } else {
            mr = ip::sqrt_rsqrt_n(fma(q[0] * q[0], C.dc[2], fma(q[1] * q[1], C.dc[3], q[2] * q[2] * C.dc[4])), im);
        }
        const double u = mr * C.dc[1], u1 = 1. + u;
        const double f = C.dc[0] * im * (im * im) * fma(-u, rcp_f(u1), log_f(u1));
        if (type == GX_POT_SPHERICALNFW) {
            d.F += f;
            return;
        }
        d.aniso = true;
        d.A[0] = fma(f, C.dc[2], d.A[0]);
        d.A[1] = fma(f, C.dc[3], d.A[1]);
        d.A[2] = fma(f, C.dc[4], d.A[2]);
        return;
    }
    default:
        d.F = __longlong_as_double(0x7ff8000000000000LL);
        return;
    }
#undef P
}

template <bool SCF, typename PV>
__device__ __forceinline__ void potential_gradient_ft(const PV &pot, const double *q, double *g) {
    Diag d;
    d.init(q);
    double gs[3] = {0., 0., 0.};  // shifted or rotated components and SCF
    bool extra = false;
    for (int i = 0; i < pot.ncomp; i++) {
        const DevComp &c = pot.c[i];
        if constexpr (SCF) {
            if (c.type == GX_POT_SCF && c.do_sr == 0) {
                scf_gradient_dev(pot.pdev + c.poff, q, gs);
                extra = true;
                continue;
            }
        }
        if (c.do_sr == 0) {
            comp_gradient_f(pot, i, q, d);
        } else {
            double qt[3], gt[3] = {0., 0., 0.};
            shift_rotate(c, q, qt);
            if constexpr (SCF) {
                if (c.type == GX_POT_SCF) scf_gradient_dev(pot.pdev + c.poff, qt, gt);
            }
            if (c.type != GX_POT_SCF) {
                Diag dt;
                dt.init(qt);
                comp_gradient_f(pot, i, qt, dt);
                dt.gradient(qt, gt);
            }
            gs[0] += fma(c.R[0], gt[0], fma(c.R[3], gt[1], c.R[6] * gt[2]));
            gs[1] += fma(c.R[1], gt[0], fma(c.R[4], gt[1], c.R[7] * gt[2]));
            gs[2] += fma(c.R[2], gt[0], fma(c.R[5], gt[1], c.R[8] * gt[2]));
            extra = true;
        }
    }
    d.gradient(q, g);
    if (extra)
        for (int k = 0; k < 3; k++) g[k] += gs[k];
}

// Gradient of a disk-bulge-halo composite (DevPot::d) in one straight run: 29 FP64
// instructions, and the two square roots, the inverse root, the three reciprocals
// and the logarithm on the integer pipe side by side instead of one after the
// other behind the component loop's branches (with it the DOP853 population of 20,011
// orbits x 1 Gyr takes 86 ms, without 134).  False where an argument is outside the integer forms' range (a point
// within 2^-6 r_s of the centre, a non-finite position): the general form then
// serves.
__device__ __forceinline__ bool dbh_gradient(const DevPot &pot, const double *q, double *g) {
    const double xy2 = fma(q[0], q[0], q[1] * q[1]);
    const double r2 = fma(q[2], q[2], xy2);
    const double w = fma(q[2], q[2], pot.d.b2);
    double ir, isz;
    const double r = ip::sqrt_rsqrt_u(r2, ir), sz = ip::sqrt_rsqrt_u(w, isz);
    const double d1 = r + pot.d.c1, d2 = r + pot.d.c2;
    const double u = r * pot.d.irs, u1 = 1. + u;
    const double zd = pot.d.a + sz;
    const double W = fma(zd, zd, xy2);
    const bool ok = ip::ok_sqrt(r2) & ip::ok_sqrt(w) & ip::ok_rcp(d1) & ip::ok_rcp(d2) & ip::ok_sqrt(W) & ip::ln_range(u1) &
                    ip::ok_rcp(u1);
    const double iW = ip::rsqrt_u(W);
    const double t1 = ip::rcp_u(d1), t2 = ip::rcp_u(d2), iu = ip::rcp_u(u1);
    const double L = ip::ln_n(u1);
    // spheres and halo share a factor 1 / r: G m / (r + c)^2 and G m (L - u / (1 + u)) / r^2
    const double s = fma(pot.d.gmh * (ir * ir), fma(-u, iu, L), fma(pot.d.gm1, t1 * t1, pot.d.gm2 * (t2 * t2)));
    const double f = pot.d.gmd * iW * (iW * iW);
    const double F = fma(ir, s, f);
    g[0] = F * q[0];
    g[1] = F * q[1];
    g[2] = fma(f, pot.d.a * isz, F) * q[2];
    return ok;
}

// A large composite (device component table) takes gala's own expressions: the
// lean forms' ulp-level differences, summed over hundreds of components, would
// exceed the 1e-12 orbit parity that DOP853 holds with a few components.
template <bool SCF>
__device__ __forceinline__ void potential_gradient_f(const DevPot &pot, const double *q, double *g) {
    if (pot.cdev) {
        potential_gradient_t<SCF, false>(table_view(pot), q, g);
        return;
    }
    if constexpr (!SCF) {
        if (pot.dbh && dbh_gradient(pot, q, g)) return;
    }
    potential_gradient_ft<SCF>(pot, q, g);
}

// Acceleration in a static frame.
template <bool SCF>
__device__ __noinline__ V3 accel_call_f(const DevPot &pot, V3 q) {
    double g[3];
    potential_gradient_f<SCF>(pot, q.v, g);
    V3 a;
    for (int c = 0; c < 3; c++) a.v[c] = -g[c];
    return a;
}

// Hamilton's equations (hamiltonian_rhs in gx_device.cuh) with the fast force.
template <bool SCF>
__device__ __noinline__ V6 rhs_call_f(const DevPot &pot, const DevFrame &fr, V6 w) {
    double g[3];
    potential_gradient_f<SCF>(pot, w.v, g);
    V6 f;
    if (fr.type == GX_FRAME_STATIC) {
        f.v[0] = w.v[3];
        f.v[1] = w.v[4];
        f.v[2] = w.v[5];
        f.v[3] = -g[0];
        f.v[4] = -g[1];
        f.v[5] = -g[2];
    } else {
        const double *O = fr.O;
        f.v[0] = w.v[3] - fma(O[1], w.v[2], -O[2] * w.v[1]);
        f.v[1] = w.v[4] - fma(-O[0], w.v[2], O[2] * w.v[0]);
        f.v[2] = w.v[5] - fma(O[0], w.v[1], -O[1] * w.v[0]);
        f.v[3] = -(g[0] + fma(O[1], w.v[5], -O[2] * w.v[4]));
        f.v[4] = -(g[1] + fma(-O[0], w.v[5], O[2] * w.v[3]));
        f.v[5] = -(g[2] + fma(O[0], w.v[4], -O[1] * w.v[3]));
    }
    return f;
}

}  // namespace fast
}  // namespace gx
