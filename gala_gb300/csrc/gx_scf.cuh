// gx_scf.cuh -- SCF basis-function expansion on the device (FP64).
//
// Same expansion as gala's scf_potential_helper / scf_gradient_helper /
// scf_density_helper (src/gala/potential/scf/src/bfe.cpp:16-189) and
// phi_nl / rho_nl / sph_grad_phi_nlm (bfe_helper.cpp:14-90), with gala's
// coefficient packing p = [G, nmax, lmax, M, r_s, S[n][l][m], T[n][l][m]].
//
// gala calls GSL once per (n, l, m) term.  Here the sums are turned round so that
// a term costs two multiply-adds for the value and four for the gradient, and
// everything else is formed once per (l, m), per l or per point:
//
//   Phi = -G M / r_s sum_l u_l sum_m N_lm P_lm(X) (fS_lm cos m phi + fT_lm sin m phi),
//   fS_lm = sum_n S_nlm C_n(xi),  u_l = s^l / (1 + s)^(2 l + 1),
//   N_lm = sqrt((2 l + 1) (l - m)! / (l + m)!)  (4 pi cancels between rho_nl and Y_lm)
//
// and the radial derivative needs the same sums over C_{n-1}^{a+1}.  The special
// functions are three-term recurrences with tabulated coefficients
// (gx_scf_table.cuh), so no division, root, power or angle is left inside:
//   Gegenbauer  C_n^a = c1 x C_{n-1}^a - c2 C_{n-2}^a, a = 2 l + 3/2,
//               C_n^{a+1} = C_{n-2}^{a+1} + (n + a) / a C_n^a
//   Legendre    (l - m) P_l^m = x (2l - 1) P_{l-1}^m - (l + m - 1) P_{l-2}^m,
//               P_m^m = (-1)^m (2m - 1)!! (1 - x^2)^{m/2}   (Condon-Shortley, as GSL)
//   cos m phi, sin m phi by the addition theorem from x / R and y / R;
//   sin theta = R / r (gala's sqrt(1 - X^2) loses digits near the pole).
// What bounds it is the FP64 pipe: per gradient 4 multiply-adds per (n, l, m), about
// 3,800 FP64 instructions at nmax = 12, lmax = 8.  131,101 points, potential and
// gradient, to host arrays: 1.5 ms (34.4 ms when each term formed its own norm,
// powers and quotients).  As in gala a term whose S and T are both zero is left
// out, so that a non-finite factor (on the pole, say) does not reach it, and at the
// centre, where every term of the density is infinite, they are summed one by one:
// terms of both signs make it NaN.
#pragma once

#include "gx_device.cuh"
#include "gx_scf_table.cuh"

namespace gx {

constexpr int SCF_MAX_N = 24;   // nmax + 1
constexpr int SCF_MAX_L = 16;   // lmax + 1

// The density where s is 0: gala's sum of its terms there, each infinite for l = 0
// (C_n^{3/2}(-1) alternates in sign) and 0 / 0 for the others, so infinite only where
// every term has one sign.
static __device__ __noinline__ double scf_density_centre(const double *p, int nmax, int lmax) {
    const double inf = __longlong_as_double(0x7ff0000000000000LL);
    const int sn = (lmax + 1) * (lmax + 1);
    double acc = 0.;
    for (int n = 0; n <= nmax; n++)
        for (int l = 0; l <= lmax; l++)
            for (int m = 0; m <= l; m++) {
                const int i = 5 + n * sn + m + (lmax + 1) * l;
                const double S = p[i], T = p[i + (nmax + 1) * sn];
                if (S == 0. && T == 0.) continue;
                acc += l == 0 ? (S + 0. * T) * (n & 1 ? -inf : inf) : inf - inf;
            }
    return acc * p[3];
}

// kind 0: value, 1: gradient (accumulated into g), 2: density.
template <int KIND>
__device__ __forceinline__ double scf_eval(const double *p, const double *q, double *g) {
    const double PI = 3.14159265358979323846;
    const double GM = p[0] * p[3];
    const int nmax = (int)p[1];
    const int lmax = (int)p[2];
    const double r_s = p[4];
    const int sn = (lmax + 1) * (lmax + 1);  // coefficients per n
    const double *Snlm = p + 5;
    const double *Tnlm = p + 5 + (nmax + 1) * sn;

    const double R2 = fma(q[0], q[0], q[1] * q[1]);
    const double R = dsqrt(R2), r = dsqrt(fma(q[2], q[2], R2));
    const double ir = ddiv(1.0, r);
    const double s = ddiv(r, r_s), s1 = 1.0 + s;
    const double X = q[2] * ir, st = R * ir;
    const double i1 = ddiv(1.0, s1);
    const double xi = (s - 1.0) * i1;
    double cp, sp;
    if (R2 > 0x1p-900) {
        const double iR = ddiv(1.0, R);
        cp = q[0] * iR;
        sp = q[1] * iR;
    } else {  // R2 has lost digits or underflowed: the angle from the coordinates scaled up
        const double x = q[0] * 0x1p600, y = q[1] * 0x1p600, Rs = sqrt(fma(x, x, y * y));
        cp = Rs == 0. ? 1. : x / Rs;  // atan2(0, 0) = 0
        sp = Rs == 0. ? 0. : y / Rs;
    }
    if (KIND == 2 && s == 0.) return scf_density_centre(p, nmax, lmax);

    double C[SCF_MAX_N], D[SCF_MAX_N];                       // C_n^a, C_{n-1}^{a+1}
    double Pl[SCF_MAX_L], Pl1[SCF_MAX_L], Pl2[SCF_MAX_L];    // P_l^m of this l and the two before
    double cm[SCF_MAX_L], sm[SCF_MAX_L];
    cm[0] = 1.;
    sm[0] = 0.;
    for (int m = 1; m <= lmax; m++) {
        cm[m] = fma(cm[m - 1], cp, -(sm[m - 1] * sp));
        sm[m] = fma(sm[m - 1], cp, cm[m - 1] * sp);
    }

    const double us = s * i1 * i1;  // u_{l+1} / u_l
    double u = i1;                  // s^l / (1 + s)^(2 l + 1)
    double acc0 = 0., acc1 = 0., acc2 = 0.;
    bool angular = false, any = false;

    for (int l = 0; l <= lmax; l++) {
        // Legendre
        if (l == 0) {
            Pl[0] = 1.;
        } else {
            for (int m = 0; m < l; m++) {
                Pl2[m] = Pl1[m];
                Pl1[m] = Pl[m];
            }
            const double x2 = X * scf::INT[2 * l - 1];
            for (int m = 0; m < l - 1; m++)
                Pl[m] = fma(x2, Pl1[m], -(scf::INT[l + m - 1] * Pl2[m])) * scf::INV[l - m];
            Pl[l - 1] = x2 * Pl1[l - 1];
            Pl[l] = -scf::INT[2 * l - 1] * st * Pl1[l - 1];
        }
        // Gegenbauer (for the density, times K_nl)
        C[0] = 1.;
        D[0] = 0.;
        if (nmax >= 1) {
            C[1] = scf::GEG1[l][1] * xi;
            D[1] = 1.;
        }
        for (int n = 2; n <= nmax; n++) {
            C[n] = fma(scf::GEG1[l][n] * xi, C[n - 1], -(scf::GEG2[l][n] * C[n - 2]));
            if (KIND == 1) D[n] = fma(scf::GEGD[l][n - 1], C[n - 1], D[n - 2]);
        }
        if (KIND == 2)
            for (int n = 0; n <= nmax; n++)
                C[n] *= 0.5 * n * (n + 4 * l + 3) + (l + 1) * (2 * l + 1);

        // sums over n, then over m
        double fr = 0., fd = 0., ft = 0., fp = 0.;
        bool anyl = false;
        for (int m = 0; m <= l; m++) {
            double sc = 0., tc = 0., sd = 0., td = 0.;
            long long nz = 0;
            const double *Sp = Snlm + (m + (lmax + 1) * l), *Tp = Tnlm + (m + (lmax + 1) * l);
#pragma unroll 4
            for (int n = 0; n <= nmax; n++) {
                const double S = __ldg(Sp + n * sn), T = __ldg(Tp + n * sn);
                const long long b = (__double_as_longlong(S) | __double_as_longlong(T)) << 1;
                nz |= b;
                const double c = b ? C[n] : 0., d = b ? D[n] : 0.;
                sc = fma(S, c, sc);
                tc = fma(T, c, tc);
                if (KIND == 1) {
                    sd = fma(S, d, sd);
                    td = fma(T, d, td);
                }
            }
            if (nz == 0) continue;
            anyl = true;
            const double np = scf::YNORM[l][m] * Pl[m];
            const double fc = fma(sc, cm[m], tc * sm[m]);
            fr = fma(np, fc, fr);
            if (KIND == 1) {
                fd = fma(np, fma(sd, cm[m], td * sm[m]), fd);
                if (l > 0) {
                    const double dp = fma(scf::INT[l] * X, Pl[m], m < l ? -(scf::INT[l + m] * Pl1[m]) : 0.);
                    ft = fma(scf::YNORM[l][m] * dp, fc, ft);
                }
                if (m > 0) fp = fma(scf::INT[m] * np, fma(tc, cm[m], -(sc * sm[m])), fp);
            }
        }
        if (anyl) {
            any = true;
            if (KIND == 0) acc0 = fma(-u, fr, acc0);
            if (KIND == 2) acc0 = fma(u, fr, acc0);
            if (KIND == 1) {
                // u s^-1 (1 + s)^-2 [(1 + s)(l (s - 1) + s) C - 2 (4 l + 3) s D]
                const double k = ddiv(u * i1 * i1, s);
                const double a = s1 * fma(scf::INT[l], s - 1.0, s), b = -2.0 * (4 * l + 3) * s;
                acc0 = fma(k, fma(a, fr, b * fd), acc0);
                if (l > 0) {
                    angular = true;
                    acc1 = fma(-u, ft, acc1);
                    acc2 = fma(-u, fp, acc2);
                }
            }
        }
        u *= us;
    }

    if (KIND == 0) return ddiv(acc0 * GM, r_s);
    if (KIND == 2) {
        // K_nl / (2 pi) s^l / (s (1 + s)^(2 l + 3))
        return any ? ddiv(acc0 * i1 * i1 * p[3], 2 * PI * s * (r_s * r_s * r_s)) : 0.;
    }
    if (!any) return 0.;
    // the theta and phi parts over s sin theta; without terms of l > 0 gala forms
    // no quotient for the first and 0 / (s sin theta) for the second
    const double iss = ddiv(1.0, s * st);
    acc1 = angular ? acc1 * iss : 0.;
    acc2 = acc2 * iss;
    const double f = ddiv(GM, r_s * r_s);
    g[0] += f * (fma(st * cp, acc0, X * cp * acc1) - sp * acc2);
    g[1] += f * (fma(st * sp, acc0, X * sp * acc1) + cp * acc2);
    g[2] += f * fma(X, acc0, -(st * acc1));
    return 0.;
}

static __device__ __noinline__ double scf_value_dev(const double *p, const double *q) { return scf_eval<0>(p, q, nullptr); }
static __device__ __noinline__ void scf_gradient_dev(const double *p, const double *q, double *g) { scf_eval<1>(p, q, g); }
static __device__ __noinline__ double scf_density_dev(const double *p, const double *q) { return scf_eval<2>(p, q, nullptr); }

}  // namespace gx
