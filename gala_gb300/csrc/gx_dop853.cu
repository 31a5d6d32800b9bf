// gx_dop853.cu -- FP64 DOP853 with gala's batch semantics.
//
// gala integrates `nbatch` orbits (default 100) as ONE ODE system of size
// n = 6 * nb: one shared step size, one RMS error norm over all 6 * nb
// components, one accept/reject decision, one dense-output grid
// (dop853.pyx:228-245 -> dop853_helper :90-193 -> dopcor, dopri/dop853.cpp:89-650).
// Static frames take dop853_static_kernel below (a batch is a cluster of one-warp
// CTAs), few orbits gx_dop853_axis.cu.  In the general kernel (rotating frames, small
// or very large batches) a batch is a group of consecutive threads of a CTA -- two
// batches per CTA when that fills the warps better (100 orbits alone leave 28 idle
// lanes), the two stepping in lock-step -- and each thread owns one orbit's six
// components:
//   * the twelve stages, FSAL evaluation and the three dense-output stages are
//     evaluated per thread in registers with gala's expression order;
//   * the error norms (err, err2) and the stiffness sums (stnum, stden) are
//     per-batch sums: a fixed-order warp butterfly plus an ordered sum over
//     warps, so the step-size sequence is deterministic run to run;
//   * every scalar of the step-size controller (x, h, facold, reject, last,
//     naccpt, ...) is computed identically by all threads of a batch from the
//     same sums, so control flow is uniform inside a batch; every thread of
//     the CTA takes part in each step's two reductions, and a CTA leaves its
//     loop when none of its batches is stepping;
//   * dense output (contd8_threadsafe, :869-904) is written directly into the
//     (6, n_out, N) result for every requested time inside [xold, xold + h].
// The loop is bounded by nmax like gala's; no thread ever waits on another CTA.
#include "gx_dop853.cuh"
#include "gx_scf.cuh"
#include "gx_dop853_tableau.cuh"
#include "gx_dop853_nystrom.cuh"
#include "gx_fast64.cuh"

namespace gx {

constexpr int DOP_MAX_WARPS = 32;

// Deterministic sums of two values over each batch of the CTA (BPC batches;
// bl is the caller's batch): a fixed-order warp butterfly, with the lanes of
// the other batch contributing zeros, then an ordered sum over warps.  Every
// thread of a batch returns the same bits.
template <int BPC>
__device__ __forceinline__ void block_sum2(double &a, double &b, double *red, int bl) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    double v[2 * BPC];
#pragma unroll
    for (int q = 0; q < BPC; q++) {
        v[q] = (bl == q) ? a : 0.0;
        v[BPC + q] = (bl == q) ? b : 0.0;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int q = 0; q < 2 * BPC; q++) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
    if (lane == 0)
#pragma unroll
        for (int q = 0; q < 2 * BPC; q++) red[q * DOP_MAX_WARPS + wid] = v[q];
    __syncthreads();
    double sa = 0., sb = 0.;
    for (int w = 0; w < nw; w++) {
        sa += red[bl * DOP_MAX_WARPS + w];
        sb += red[(BPC + bl) * DOP_MAX_WARPS + w];
    }
    __syncthreads();
    a = sa;
    b = sb;
}

#define RHS(yin, kout)                                                   \
    do {                                                                 \
        if (active) {                                                    \
            V6 a_;                                                       \
            for (int c_ = 0; c_ < 6; c_++) a_.v[c_] = yin[c_];           \
            const V6 r_ = fast::rhs_call_f<SCF>(pot, fr, a_);            \
            for (int c_ = 0; c_ < 6; c_++) kout[c_] = r_.v[c_];          \
        } else {                                                         \
            for (int c_ = 0; c_ < 6; c_++) kout[c_] = 0.;                \
        }                                                                \
    } while (0)

template <int MAXT, bool SCF, int BPC>
__global__ void __launch_bounds__(MAXT, 1)
dop853_kernel(const __grid_constant__ DevPot pot, const __grid_constant__ DevFrame fr, DopArgs A,
              const double *__restrict__ w0, int64_t n, const double *__restrict__ t, double *__restrict__ out,
              int32_t *__restrict__ status,
              int64_t *__restrict__ stats) {
    using namespace dop;
    __shared__ double red[4 * DOP_MAX_WARPS];
    // a CTA that starts after cancellation integrates nothing (one reader, CTA-uniform)
    if (__syncthreads_or(threadIdx.x == 0 && cancel_requested(A.cancel))) return;

    // BPC batches per CTA, batch bl on threads [bl * nbatch, (bl + 1) * nbatch)
    const int nbs = A.nbatch;
    const int bl = (BPC == 1) ? 0 : min((int)threadIdx.x / nbs, BPC - 1);
    const int j = threadIdx.x - bl * nbs;  // lane within the batch
    const int64_t b = (int64_t)blockIdx.x * BPC + bl;
    const int64_t nbt = (n + nbs - 1) / nbs;
    const bool batch_ok = b < nbt && j < nbs;
    const int64_t i0 = b * nbs;
    const int nb = batch_ok ? (int)((i0 + nbs <= n) ? nbs : n - i0) : 0;
    const bool active = batch_ok && j < nb;
    const int nsys = 6 * nb;

    double y[6], k1[6], k2[6], k3[6], k4[6], k5[6], k6[6], k7[6], k8[6], k9[6], k10[6], yy1[6];
    for (int c = 0; c < 6; c++) y[c] = active ? w0[c * n + i0 + j] : 0.;

    // dop853() front-end defaults with dop853_helper's arguments (dop853.pyx:157-182)
    double x = t[0];
    const double xend = t[A.ntimes - 1];
    double h = t[1] - t[0];
    double hmax = A.dt_max;
    const double uround = 2.220446049250313e-16;
    const double safe = 0.9, fac1 = 0.333, fac2 = 6.0;  // and beta = 0
    int64_t nmax = A.nmax, nstiff = A.nstiff;
    if (!nmax) nmax = 1000000;
    if (!nstiff) nstiff = 1000;
    else if (nstiff < 0) nstiff = nmax + 10;
    if (hmax == 0.0) hmax = xend - x;

    double facold = 1.0E-4;
    const double facc1 = 1.0 / fac1, facc2 = 1.0 / fac2;
    const double posneg = sign_d(1.0, xend - x);
    const double atoli = A.atol, rtoli = A.rtol;
    int last = 0, reject = 0, iasti = 0, nonsti = 0, idid = 0;
    double hlamb = 0.0;
    int64_t nfcn = 0, nstep = 0, naccpt = 0, nrejct = 0;
    int64_t out_idx = 0, out_slot = 0;

    RHS(y, k1);
    hmax = fabs(hmax);
    if (h == 0.0) {
        // hinit (dop853.cpp:18-86), scalar tolerances, CTA-wide norms
        double dnf = 0.0, dny = 0.0;
        for (int c = 0; c < 6; c++) {
            const double sk = atoli + rtoli * fabs(y[c]);
            double sqr = k1[c] / sk;
            dnf += active ? sqr * sqr : 0.;
            sqr = y[c] / sk;
            dny += active ? sqr * sqr : 0.;
        }
        block_sum2<BPC>(dnf, dny, red, bl);
        double hh = ((dnf <= 1.0E-10) || (dny <= 1.0E-10)) ? 1.0E-6 : sqrt(dny / dnf) * 0.01;
        hh = min_d(hh, hmax);
        hh = sign_d(hh, posneg);
        for (int c = 0; c < 6; c++) yy1[c] = y[c] + hh * k1[c];
        RHS(yy1, k2);
        double der2 = 0.0, unused = 0.0;
        for (int c = 0; c < 6; c++) {
            const double sk = atoli + rtoli * fabs(y[c]);
            const double sqr = (k2[c] - k1[c]) / sk;
            der2 += active ? sqr * sqr : 0.;
        }
        block_sum2<BPC>(der2, unused, red, bl);
        der2 = sqrt(der2) / hh;
        const double der12 = max_d(fabs(der2), sqrt(dnf));
        const double h1 = (der12 <= 1.0E-15) ? max_d(1.0E-6, fabs(hh) * 1.0E-3) : pow(0.01 / der12, 1.0 / 8.0);
        hh = min_d(100.0 * fabs(hh), min_d(h1, hmax));
        h = sign_d(hh, posneg);
    }
    nfcn += 2;

    bool done = !batch_ok;
    double xold = 0.0, hout = 0.0, xph = 0.0;
    for (;;) {
        // the batches of a CTA step in lock-step: every thread takes part in the
        // two CTA reductions of each step, and the loop ends when no batch of
        // the CTA is stepping any more
        if (!__syncthreads_or(done ? 0 : 1)) break;
        bool stepping = !done;
        if (stepping && h != h) nan_steps(nmax, naccpt, nstep, nfcn, nrejct);
        if (stepping && nstep > nmax) {
            idid = -2;
            done = true;
            stepping = false;
        }
        if (stepping && 0.1 * fabs(h) <= fabs(x) * uround) {
            idid = -3;
            done = true;
            stepping = false;
        }
        if (stepping) {
            if ((x + 1.01 * h - xend) * posneg > 0.0) {
                h = xend - x;
                last = 1;
            }
            xold = x;
            hout = h;
            nstep++;

            // the twelve stages (dop853.cpp:368-414)
            // stage sums as fused multiply-add chains in gala's term order
            for (int c = 0; c < 6; c++) yy1[c] = fma(h * a21, k1[c], y[c]);
            RHS(yy1, k2);
            for (int c = 0; c < 6; c++) yy1[c] = fma(h, fma(a32, k2[c], a31 * k1[c]), y[c]);
            RHS(yy1, k3);
            for (int c = 0; c < 6; c++) yy1[c] = fma(h, fma(a43, k3[c], a41 * k1[c]), y[c]);
            RHS(yy1, k4);
            for (int c = 0; c < 6; c++) yy1[c] = fma(h, fma(a54, k4[c], fma(a53, k3[c], a51 * k1[c])), y[c]);
            RHS(yy1, k5);
            for (int c = 0; c < 6; c++) yy1[c] = fma(h, fma(a65, k5[c], fma(a64, k4[c], a61 * k1[c])), y[c]);
            RHS(yy1, k6);
            for (int c = 0; c < 6; c++)
                yy1[c] = fma(h, fma(a76, k6[c], fma(a75, k5[c], fma(a74, k4[c], a71 * k1[c]))), y[c]);
            RHS(yy1, k7);
            for (int c = 0; c < 6; c++)
                yy1[c] = fma(h, fma(a87, k7[c], fma(a86, k6[c], fma(a85, k5[c], fma(a84, k4[c], a81 * k1[c])))), y[c]);
            RHS(yy1, k8);
            for (int c = 0; c < 6; c++)
                yy1[c] = fma(h, fma(a98, k8[c], fma(a97, k7[c], fma(a96, k6[c], fma(a95, k5[c], fma(a94, k4[c],
                                                                                                    a91 * k1[c]))))),
                             y[c]);
            RHS(yy1, k9);
            for (int c = 0; c < 6; c++)
                yy1[c] = fma(h, fma(a109, k9[c], fma(a108, k8[c], fma(a107, k7[c], fma(a106, k6[c], fma(a105, k5[c],
                                    fma(a104, k4[c], a101 * k1[c])))))), y[c]);
            RHS(yy1, k10);
            for (int c = 0; c < 6; c++)
                yy1[c] = fma(h, fma(a1110, k10[c], fma(a119, k9[c], fma(a118, k8[c], fma(a117, k7[c], fma(a116, k6[c],
                                    fma(a115, k5[c], fma(a114, k4[c], a111 * k1[c]))))))), y[c]);
            RHS(yy1, k2);
            xph = x + h;
            for (int c = 0; c < 6; c++)
                yy1[c] = fma(h, fma(a1211, k2[c], fma(a1210, k10[c], fma(a129, k9[c], fma(a128, k8[c], fma(a127, k7[c],
                                    fma(a126, k6[c], fma(a125, k5[c], fma(a124, k4[c], a121 * k1[c])))))))), y[c]);
            RHS(yy1, k3);
            nfcn += 11;
            for (int c = 0; c < 6; c++) {
                k4[c] = fma(b12, k3[c], fma(b11, k2[c], fma(b10, k10[c], fma(b9, k9[c], fma(b8, k8[c], fma(b7, k7[c],
                            fma(b6, k6[c], b1 * k1[c])))))));
                k5[c] = fma(h, k4[c], y[c]);
            }
        }

        // error estimation (:416-444), summed over each batch
        double err = 0.0, err2 = 0.0;
        if (stepping && active) {
            for (int c = 0; c < 6; c++) {
                const double isk = fast::rcp_f(fma(rtoli, fmax(fabs(y[c]), fabs(k5[c])), atoli));
                double erri = fma(-bhh3, k3[c], fma(-bhh2, k9[c], fma(-bhh1, k1[c], k4[c])));
                double sqr = erri * isk;
                err2 = fma(sqr, sqr, err2);
                erri = fma(er12, k3[c], fma(er11, k2[c], fma(er10, k10[c], fma(er9, k9[c], fma(er8, k8[c],
                           fma(er7, k7[c], fma(er6, k6[c], er1 * k1[c])))))));
                sqr = erri * isk;
                err = fma(sqr, sqr, err);
            }
        }
        block_sum2<BPC>(err, err2, red, bl);
        double hnew = h, fac11 = 1.0;
        bool acc = false;
        if (stepping) {
            double deno = err + 0.01 * err2;
            if (deno <= 0.0) deno = 1.0;
            err = fabs(h) * err * sqrt(1.0 / (deno * (double)nsys));
            // computation of hnew (:446-452); gala's pow(err, expo1) with expo1 = 1/8
            // (beta = 0) as three square roots instead of pow's ~84 FP64-pipe instructions
            fac11 = sqrt(sqrt(sqrt(err)));
            double fac = fac11;  // gala divides by pow(facold, beta) == 1 for its beta = 0
            fac = max_d(facc2, min_d(facc1, fac / safe));
            hnew = h / fac;
            acc = err <= 1.0;
            if (acc) {
                facold = max_d(err, 1.0E-4);
                naccpt++;
                RHS(k5, k4);
                nfcn++;
            }
        }

        // stiffness detection (:463-486); like gala, the first detection returns -4.
        // The sums are formed every step (zero where no test is due) so that all
        // batches of the CTA share the barrier.
        const bool stiff_due = stepping && acc && (!(naccpt % nstiff) || (iasti > 0));
        double stnum = 0.0, stden = 0.0;
        if (stiff_due && active) {
            for (int c = 0; c < 6; c++) {
                double sqr = k4[c] - k3[c];
                stnum += sqr * sqr;
                sqr = k5[c] - yy1[c];
                stden += sqr * sqr;
            }
        }
        block_sum2<BPC>(stnum, stden, red, bl);
        if (stiff_due) {
            if (stden > 0.0) hlamb = h * sqrt(stnum / stden);
            if (hlamb > 6.1) {
                nonsti = 0;
                iasti++;
                idid = -4;
                done = true;
                stepping = false;
            } else {
                nonsti++;
                if (nonsti == 6) iasti = 0;
            }
        }

        if (stepping && acc) {
            // Output times inside [xold, xold + hout] (:584-612): [out_idx, out_end).
            // Only every out_stride-th time is stored; the three dense-output stages
            // are evaluated only for a step that holds a stored time (their results
            // feed nothing else: the next step starts from k4 = f(k5) and recomputes
            // every other stage), so the trajectory is unchanged.
            int64_t out_end = out_idx, first_kept = 0;
            if (A.save_all) {
                const double x0 = xold, x1 = x0 + hout;
                while (out_end < A.ntimes) {
                    const double t_out = t[out_end];
                    if (!((x0 <= t_out && t_out <= x1) || (x1 <= t_out && t_out <= x0))) break;
                    out_end++;
                }
                first_kept = (out_idx + A.out_stride - 1) / A.out_stride * A.out_stride;
            }
            if (A.save_all && first_kept < out_end) {
                // dense output preparation (:492-582)
                double r5[6], r6[6], r7[6], r8[6];
#define GX_D8(p, k1_, k6_, k7_, k8_, k9_, k10_, k2_, k3_)                                                      \
    fma(p##12, k3_, fma(p##11, k2_, fma(p##10, k10_, fma(p##9, k9_, fma(p##8, k8_, fma(p##7, k7_,              \
        fma(p##6, k6_, p##1 * k1_)))))))
                for (int c = 0; c < 6; c++) {
                    r5[c] = GX_D8(d4, k1[c], k6[c], k7[c], k8[c], k9[c], k10[c], k2[c], k3[c]);
                    r6[c] = GX_D8(d5, k1[c], k6[c], k7[c], k8[c], k9[c], k10[c], k2[c], k3[c]);
                    r7[c] = GX_D8(d6, k1[c], k6[c], k7[c], k8[c], k9[c], k10[c], k2[c], k3[c]);
                    r8[c] = GX_D8(d7, k1[c], k6[c], k7[c], k8[c], k9[c], k10[c], k2[c], k3[c]);
                }
#undef GX_D8
                for (int c = 0; c < 6; c++)
                    yy1[c] = fma(h, fma(a1413, k4[c], fma(a1412, k3[c], fma(a1411, k2[c], fma(a1410, k10[c],
                                 fma(a149, k9[c], fma(a148, k8[c], fma(a147, k7[c], a141 * k1[c]))))))), y[c]);
                RHS(yy1, k10);
                for (int c = 0; c < 6; c++)
                    yy1[c] = fma(h, fma(a1514, k10[c], fma(a1513, k4[c], fma(a1512, k3[c], fma(a1511, k2[c],
                                 fma(a158, k8[c], fma(a157, k7[c], fma(a156, k6[c], a151 * k1[c]))))))), y[c]);
                RHS(yy1, k2);
                for (int c = 0; c < 6; c++)
                    yy1[c] = fma(h, fma(a1615, k2[c], fma(a1614, k10[c], fma(a1613, k4[c], fma(a169, k9[c],
                                 fma(a168, k8[c], fma(a167, k7[c], fma(a166, k6[c], a161 * k1[c]))))))), y[c]);
                RHS(yy1, k3);
                nfcn += 3;
                double r1[6], r2[6], r3[6], r4[6];
                for (int c = 0; c < 6; c++) {
                    r5[c] = h * fma(d416, k3[c], fma(d415, k2[c], fma(d414, k10[c], fma(d413, k4[c], r5[c]))));
                    r6[c] = h * fma(d516, k3[c], fma(d515, k2[c], fma(d514, k10[c], fma(d513, k4[c], r6[c]))));
                    r7[c] = h * fma(d616, k3[c], fma(d615, k2[c], fma(d614, k10[c], fma(d613, k4[c], r7[c]))));
                    r8[c] = h * fma(d716, k3[c], fma(d715, k2[c], fma(d714, k10[c], fma(d713, k4[c], r8[c]))));
                    r1[c] = y[c];
                    const double ydiff = k5[c] - y[c];
                    r2[c] = ydiff;
                    const double bspl = fma(h, k1[c], -ydiff);
                    r3[c] = bspl;
                    r4[c] = fma(-h, k4[c], ydiff) - bspl;
                }

                for (int64_t oi = first_kept; oi < out_end; oi += A.out_stride) {
                    const double s = (t[oi] - xold) / hout;
                    const double s1 = 1.0 - s;
                    if (active) {
                        for (int c = 0; c < 6; c++) {
                            const double v =
                                fma(s, fma(s1, fma(s, fma(s1, fma(s, fma(s1, fma(s, r8[c], r7[c]), r6[c]), r5[c]),
                                                          r4[c]), r3[c]), r2[c]), r1[c]);
                            __stcs(&out[((int64_t)c * A.n_out + out_slot) * n + i0 + j], v);
                        }
                    }
                    out_slot++;
                }
            }
            out_idx = out_end;


            for (int c = 0; c < 6; c++) {
                k1[c] = k4[c];
                y[c] = k5[c];
            }
            x = xph;
            if (last) {
                idid = 1;
                done = true;
            } else {
                if (fabs(hnew) > hmax) hnew = posneg * hmax;
                if (reject) hnew = posneg * min_d(fabs(hnew), fabs(h));
                reject = 0;
            }
        } else if (stepping) {
            hnew = h / min_d(facc1, fac11 / safe);
            reject = 1;
            if (naccpt >= 1) nrejct = nrejct + 1;
            last = 0;
        }
        if (stepping && !done) h = hnew;
    }
    (void)nonsti;

    if (!A.save_all && active)
        for (int c = 0; c < 6; c++) out[c * n + i0 + j] = y[c];
    if (j == 0 && batch_ok) {
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

// ---------------------------------------------------------------------------
// Static frames: x' = v, v' = a(x), so the tableau collapses (gx_dop853_nystrom.cuh)
// and a step needs the twelve accelerations only.  Against the kernel above that is
// 380 instead of 534 FP64 instructions of stage algebra per step, 72 instead of 144
// registers of derivatives, and so several warps per scheduler instead of one or two.
//
// A batch is a cluster of one-warp CTAs (100 orbits: 4), placed on as many SMs:
// the FP64 unit of an SM takes one warp instruction per 19 cycles and a warp alone
// at most one per 64, so the warps of a few batches run fastest on SMs of their own
// and many batches still fill every SM evenly (201 batches of 4 warps: 5 or 6 warps
// on each of 152 SMs; as CTAs of two batches they held 101 SMs).  The step's sums
// go through distributed shared memory: every warp writes its partial sums to each
// CTA of the cluster, one cluster barrier, and all add the partial sums in rank
// order, so all take the same decisions.
//
// Measured: 20,011 MW orbits x 1 Gyr (201 batches) 180 -> 86 ms (230 ms before the
// force left the FP64 pipe), now 823 FP64 instructions per step and warp and bound
// by the FP64 units of the SMs that hold six warps.
// ---------------------------------------------------------------------------
constexpr int NYS_MAX_WARPS = 8;

// Sums of a and b over the G warps of the batch, the same bits in every lane of
// every warp: the two halves of a warp fold one value each, then the partial sums
// are added in rank order.  buf: [2][NYS_MAX_WARPS], one of two used in turn.
__device__ __forceinline__ void nys_sum2(double &a, double &b, double (*buf)[NYS_MAX_WARPS], int G, unsigned rank) {
    const int lane = threadIdx.x;
    const double oa = __shfl_xor_sync(0xffffffffu, a, 16), ob = __shfl_xor_sync(0xffffffffu, b, 16);
    double v = pick(lane < 16, a, b) + pick(lane < 16, oa, ob);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (G == 1) {
        a = __shfl_sync(0xffffffffu, v, 0);
        b = __shfl_sync(0xffffffffu, v, 16);
        return;
    }
    // lane k (a) and lane 16 + k (b) write to CTA k
    if ((lane & 15) < G) cluster_store(&buf[lane >> 4][rank], lane & 15, v);
    cluster_sync_all();
    a = buf[0][0];
    b = buf[1][0];
    for (int k = 1; k < G; k++) {
        a += buf[0][k];
        b += buf[1][k];
    }
}

template <bool SCF>
__device__ __forceinline__ void accel(const DevPot &pot, bool active, const double *x, double *k) {
    V3 r = {{0., 0., 0.}};
    if (active) {
        V3 q;
        for (int c = 0; c < 3; c++) q.v[c] = x[c];
        r = fast::accel_call_f<SCF>(pot, q);
    }
    for (int c = 0; c < 3; c++) k[c] = r.v[c];
}
#define ACC(xin, kout) accel<SCF>(pot, active, xin, kout)

template <bool SCF>
__global__ void __launch_bounds__(32, 8)
dop853_static_kernel(const __grid_constant__ DevPot pot, DopArgs A, int G, const double *__restrict__ w0, int64_t n,
                     const double *__restrict__ t, double *__restrict__ out, int32_t *__restrict__ status,
                     int64_t *__restrict__ stats) {
    using namespace dop;
    __shared__ double buf[2][2][NYS_MAX_WARPS];
    __shared__ int stop;
    const unsigned rank = G == 1 ? 0u : cluster_rank();
    const int lane = threadIdx.x;
    // a batch that starts after cancellation is not integrated: the cluster takes
    // the decision of its first CTA (buf as the message, before its first use)
    if (G == 1) {
        if (lane == 0) stop = cancel_requested(A.cancel);
        __syncwarp();
    } else {
        cluster_sync_all();  // every CTA's shared memory exists
        if (rank == 0) {
            double c = 0.;
            if (lane == 0) c = cancel_requested(A.cancel) ? 1. : 0.;
            c = __shfl_sync(0xffffffffu, c, 0);
            if (lane < G) cluster_store(&buf[0][0][0], lane, c);
        }
        cluster_sync_all();
        if (lane == 0) stop = buf[0][0][0] != 0.;
        cluster_sync_all();
    }
    if (stop) return;

    const int64_t b = blockIdx.x / G;
    const int64_t i0 = b * A.nbatch;
    const int nb = (int)min((int64_t)A.nbatch, n - i0);
    const int j = (int)rank * 32 + lane;
    const bool active = j < nb;
    const double nsys = 6 * nb;

    double x[3], v[3], xn[3], vn[3], xs[3];
    double k1[3], k2[3], k3[3], k4[3], k5[3], k6[3], k7[3], k8[3], k9[3], k10[3], k11[3], k12[3];
    for (int c = 0; c < 3; c++) {
        x[c] = active ? w0[c * n + i0 + j] : 0.;
        v[c] = active ? w0[(3 + c) * n + i0 + j] : 0.;
    }

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

    ACC(x, k1);
    hmax = fabs(hmax);
    if (h == 0.0) {
        // hinit (dop853.cpp:18-86), scalar tolerances, batch-wide norms
        double dnf = 0.0, dny = 0.0;
        for (int c = 0; c < 3; c++) {
            const double skx = atoli + rtoli * fabs(x[c]), skv = atoli + rtoli * fabs(v[c]);
            double q = ddiv(v[c], skx), p = ddiv(k1[c], skv);
            dnf += active ? q * q + p * p : 0.;
            q = ddiv(x[c], skx);
            p = ddiv(v[c], skv);
            dny += active ? q * q + p * p : 0.;
        }
        nys_sum2(dnf, dny, buf[par], G, rank);
        par ^= 1;
        double hh = ((dnf <= 1.0E-10) || (dny <= 1.0E-10)) ? 1.0E-6 : sqrt(dny / dnf) * 0.01;
        hh = min_d(hh, hmax);
        hh = sign_d(hh, posneg);
        for (int c = 0; c < 3; c++) xs[c] = x[c] + hh * v[c];
        ACC(xs, k2);
        double der2 = 0.0, unused = 0.0;
        for (int c = 0; c < 3; c++) {
            const double skx = atoli + rtoli * fabs(x[c]), skv = atoli + rtoli * fabs(v[c]);
            const double q = ddiv(hh * k1[c], skx), p = ddiv(k2[c] - k1[c], skv);  // f(y + hh f) - f(y)
            der2 += active ? q * q + p * p : 0.;
        }
        nys_sum2(der2, unused, buf[par], G, rank);
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

        // stage positions and their accelerations
#define HV(i) fma(h, fma(h, S, nc##i * v[c]), x[c])
        for (int c = 0; c < 3; c++) xs[c] = fma(h, nc2 * v[c], x[c]);
        ACC(xs, k2);
        for (int c = 0; c < 3; c++) {
            const double S = n3_1 * k1[c];
            xs[c] = HV(3);
        }
        ACC(xs, k3);
        for (int c = 0; c < 3; c++) {
            const double S = fma(n4_2, k2[c], n4_1 * k1[c]);
            xs[c] = HV(4);
        }
        ACC(xs, k4);
        for (int c = 0; c < 3; c++) {
            const double S = fma(n5_3, k3[c], fma(n5_2, k2[c], n5_1 * k1[c]));
            xs[c] = HV(5);
        }
        ACC(xs, k5);
        for (int c = 0; c < 3; c++) {
            const double S = fma(n6_4, k4[c], fma(n6_3, k3[c], n6_1 * k1[c]));
            xs[c] = HV(6);
        }
        ACC(xs, k6);
        for (int c = 0; c < 3; c++) {
            const double S = fma(n7_5, k5[c], fma(n7_4, k4[c], fma(n7_3, k3[c], n7_1 * k1[c])));
            xs[c] = HV(7);
        }
        ACC(xs, k7);
        for (int c = 0; c < 3; c++) {
            const double S = fma(n8_6, k6[c], fma(n8_5, k5[c], fma(n8_4, k4[c], fma(n8_3, k3[c], n8_1 * k1[c]))));
            xs[c] = HV(8);
        }
        ACC(xs, k8);
        for (int c = 0; c < 3; c++) {
            const double S = fma(n9_7, k7[c], fma(n9_6, k6[c], fma(n9_5, k5[c], fma(n9_4, k4[c], fma(n9_3, k3[c],
                                 n9_1 * k1[c])))));
            xs[c] = HV(9);
        }
        ACC(xs, k9);
        for (int c = 0; c < 3; c++) {
            const double S = fma(n10_8, k8[c], fma(n10_7, k7[c], fma(n10_6, k6[c], fma(n10_5, k5[c], fma(n10_4, k4[c],
                                 fma(n10_3, k3[c], n10_1 * k1[c]))))));
            xs[c] = HV(10);
        }
        ACC(xs, k10);
        for (int c = 0; c < 3; c++) {
            const double S = fma(n11_9, k9[c], fma(n11_8, k8[c], fma(n11_7, k7[c], fma(n11_6, k6[c], fma(n11_5, k5[c],
                                 fma(n11_4, k4[c], fma(n11_3, k3[c], n11_1 * k1[c])))))));
            xs[c] = HV(11);
        }
        ACC(xs, k11);
        for (int c = 0; c < 3; c++) {
            const double S = fma(n12_10, k10[c], fma(n12_9, k9[c], fma(n12_8, k8[c], fma(n12_7, k7[c], fma(n12_6, k6[c],
                                 fma(n12_5, k5[c], fma(n12_4, k4[c], fma(n12_3, k3[c], n12_1 * k1[c]))))))));
            xs[c] = HV(12);
        }
        ACC(xs, k12);
#undef HV
        const double tph = tx + h;
        nfcn += 11;

        // the new state and the error estimates (dop853.cpp:410-444); a position's
        // estimates carry a factor h, taken into its scale
        double err = 0.0, err2 = 0.0;
        for (int c = 0; c < 3; c++) {
            const double bv = fma(b12, k12[c], fma(b11, k11[c], fma(b10, k10[c], fma(b9, k9[c], fma(b8, k8[c],
                                  fma(b7, k7[c], fma(b6, k6[c], b1 * k1[c])))))));
            const double bx = fma(nb11, k11[c], fma(nb10, k10[c], fma(nb9, k9[c], fma(nb8, k8[c], fma(nb7, k7[c],
                                  fma(nb6, k6[c], nb1 * k1[c]))))));
            vn[c] = fma(h, bv, v[c]);
            xn[c] = fma(h, fma(h, bx, v[c]), x[c]);
            const double iskx = h * fast::rcp_f(fma(rtoli, max_abs(x[c], xn[c]), atoli));
            const double iskv = fast::rcp_f(fma(rtoli, max_abs(v[c], vn[c]), atoli));
            const double hx = fma(nbh11, k11[c], fma(nbh10, k10[c], fma(nbh9, k9[c], fma(nbh8, k8[c], fma(nbh7, k7[c],
                                  fma(nbh6, k6[c], fma(nbh5, k5[c], fma(nbh4, k4[c], nbh1 * k1[c]))))))));
            const double hv = fma(-bhh3, k12[c], fma(-bhh2, k9[c], fma(-bhh1, k1[c], bv)));
            double q = hx * iskx;
            err2 = fma(q, q, err2);
            q = hv * iskv;
            err2 = fma(q, q, err2);
            const double ex = fma(ner11, k11[c], fma(ner10, k10[c], fma(ner9, k9[c], fma(ner8, k8[c], fma(ner7, k7[c],
                                  fma(ner6, k6[c], fma(ner5, k5[c], fma(ner4, k4[c], ner1 * k1[c]))))))));
            const double ev = fma(er12, k12[c], fma(er11, k11[c], fma(er10, k10[c], fma(er9, k9[c], fma(er8, k8[c],
                                  fma(er7, k7[c], fma(er6, k6[c], er1 * k1[c])))))));
            q = ex * iskx;
            err = fma(q, q, err);
            q = ev * iskv;
            err = fma(q, q, err);
        }
        if (!active) err = err2 = 0.0;
        nys_sum2(err, err2, buf[par], G, rank);
        par ^= 1;
        double deno = fma(0.01, err2, err);
        // gala's deno <= 0, and where its reciprocal would overflow: the estimates hold nothing but
        // accelerations (no rounding of the velocities), so nearly free orbits come that low
        if (deno < 0x1p-1000) deno = 1.0;
        err = fabs(h) * err * dsqrt(ddiv(1.0, deno * nsys));
        // computation of hnew (:446-452); gala's pow(err, 1/8) (beta = 0) as three square roots
        const double fac11 = dsqrt(dsqrt(dsqrt(err)));
        const double fac = max_d(facc2, min_d(facc1, ddiv(fac11, safe)));
        double hnew = ddiv(h, fac);
        if (err <= 1.0) {
            naccpt++;
            double kn[3];
            ACC(xn, kn);
            nfcn++;

            // stiffness detection (:463-486); like gala, the first detection returns -4.
            // The last stage's velocity is formed only here.
            bool stiff = false;
            const bool due = --to_test == 0;
            if (due) to_test = nstiff;
            if (due || (iasti > 0)) {
                double stnum = 0.0, stden = 0.0;
                for (int c = 0; c < 3; c++) {
                    const double v12 = fma(h, fma(a1211, k11[c], fma(a1210, k10[c], fma(a129, k9[c], fma(a128, k8[c],
                                           fma(a127, k7[c], fma(a126, k6[c], fma(a125, k5[c], fma(a124, k4[c],
                                           a121 * k1[c])))))))), v[c]);
                    double q = vn[c] - v12;
                    stnum = fma(q, q, stnum);
                    stden = fma(q, q, stden);
                    q = kn[c] - k12[c];
                    stnum = fma(q, q, stnum);
                    q = xn[c] - xs[c];
                    stden = fma(q, q, stden);
                }
                if (!active) stnum = stden = 0.0;
                nys_sum2(stnum, stden, buf[par], G, rank);
                par ^= 1;
                if (stden > 0.0) hlamb = h * dsqrt(ddiv(stnum, stden));
                if (hlamb > 6.1) {
                    nonsti = 0;
                    iasti++;
                    idid = -4;
                    stiff = true;
                } else {
                    nonsti++;
                    if (nonsti == 6) iasti = 0;
                }
            }
            if (stiff) break;

            // output times inside [xold, xold + hout] (see the kernel above)
            int64_t out_end = out_idx;
            if (A.save_all) {
                const double x0 = xold, x1 = x0 + hout;
                while (out_end < A.ntimes) {
                    const double t_out = t[out_end];
                    if (!((x0 <= t_out && t_out <= x1) || (x1 <= t_out && t_out <= x0))) break;
                    out_end++;
                }
            }
            if (A.save_all && kept < out_end) {
                // dense output preparation (:492-582).  The stage velocities V_i (the
                // positions' derivatives) are formed here from the accelerations.
#define GX_D8(p, q1, q6, q7, q8, q9, q10, q11, q12)                                                            \
    fma(p##12, q12, fma(p##11, q11, fma(p##10, q10, fma(p##9, q9, fma(p##8, q8, fma(p##7, q7, fma(p##6, q6, p##1 * q1)))))))
                double r5[3], r6[3], r7[3], r8[3], p15[3], p16[3];
                for (int c = 0; c < 3; c++) {
                    const double V6 = fma(h, fma(a65, k5[c], fma(a64, k4[c], a61 * k1[c])), v[c]);
                    const double V7 = fma(h, fma(a76, k6[c], fma(a75, k5[c], fma(a74, k4[c], a71 * k1[c]))), v[c]);
                    const double V8 = fma(h, fma(a87, k7[c], fma(a86, k6[c], fma(a85, k5[c], fma(a84, k4[c], a81 * k1[c])))), v[c]);
                    const double V9 = fma(h, fma(a98, k8[c], fma(a97, k7[c], fma(a96, k6[c], fma(a95, k5[c], fma(a94, k4[c],
                                             a91 * k1[c]))))), v[c]);
                    const double V10 = fma(h, fma(a109, k9[c], fma(a108, k8[c], fma(a107, k7[c], fma(a106, k6[c], fma(a105, k5[c],
                                              fma(a104, k4[c], a101 * k1[c])))))), v[c]);
                    const double V11 = fma(h, fma(a1110, k10[c], fma(a119, k9[c], fma(a118, k8[c], fma(a117, k7[c],
                                              fma(a116, k6[c], fma(a115, k5[c], fma(a114, k4[c], a111 * k1[c]))))))), v[c]);
                    const double V12 = fma(h, fma(a1211, k11[c], fma(a1210, k10[c], fma(a129, k9[c], fma(a128, k8[c],
                                              fma(a127, k7[c], fma(a126, k6[c], fma(a125, k5[c], fma(a124, k4[c],
                                              a121 * k1[c])))))))), v[c]);
                    r5[c] = fma(d413, vn[c], GX_D8(d4, v[c], V6, V7, V8, V9, V10, V11, V12));
                    r6[c] = fma(d513, vn[c], GX_D8(d5, v[c], V6, V7, V8, V9, V10, V11, V12));
                    r7[c] = fma(d613, vn[c], GX_D8(d6, v[c], V6, V7, V8, V9, V10, V11, V12));
                    r8[c] = fma(d713, vn[c], GX_D8(d7, v[c], V6, V7, V8, V9, V10, V11, V12));
                    xs[c] = fma(h, fma(a1413, vn[c], fma(a1412, V12, fma(a1411, V11, fma(a1410, V10, fma(a149, V9,
                                   fma(a148, V8, fma(a147, V7, a141 * v[c]))))))), x[c]);
                    p15[c] = fma(a1513, vn[c], fma(a1512, V12, fma(a1511, V11, fma(a158, V8, fma(a157, V7, fma(a156, V6,
                                 a151 * v[c]))))));
                    p16[c] = fma(a1613, vn[c], fma(a169, V9, fma(a168, V8, fma(a167, V7, fma(a166, V6, a161 * v[c])))));
                }
                double k14[3], k15[3], k16[3], V14[3], V15[3];
                ACC(xs, k14);
                for (int c = 0; c < 3; c++) {
                    V14[c] = fma(h, fma(a1413, kn[c], fma(a1412, k12[c], fma(a1411, k11[c], fma(a1410, k10[c],
                                    fma(a149, k9[c], fma(a148, k8[c], fma(a147, k7[c], a141 * k1[c]))))))), v[c]);
                    xs[c] = fma(h, fma(a1514, V14[c], p15[c]), x[c]);
                }
                ACC(xs, k15);
                for (int c = 0; c < 3; c++) {
                    V15[c] = fma(h, fma(a1514, k14[c], fma(a1513, kn[c], fma(a1512, k12[c], fma(a1511, k11[c],
                                    fma(a158, k8[c], fma(a157, k7[c], fma(a156, k6[c], a151 * k1[c]))))))), v[c]);
                    xs[c] = fma(h, fma(a1615, V15[c], fma(a1614, V14[c], p16[c])), x[c]);
                }
                ACC(xs, k16);
                nfcn += 3;
                const int64_t rows = A.n_out * n;
                int64_t next = kept;
                for (int c = 0; c < 3; c++) {
                    const double V16 = fma(h, fma(a1615, k15[c], fma(a1614, k14[c], fma(a1613, kn[c], fma(a169, k9[c],
                                              fma(a168, k8[c], fma(a167, k7[c], fma(a166, k6[c], a161 * k1[c]))))))), v[c]);
#define GX_D3(p, base, q14, q15, q16) h * fma(p##16, q16, fma(p##15, q15, fma(p##14, q14, base)))
                    const double x5 = GX_D3(d4, r5[c], V14[c], V15[c], V16), x6 = GX_D3(d5, r6[c], V14[c], V15[c], V16);
                    const double x7 = GX_D3(d6, r7[c], V14[c], V15[c], V16), x8 = GX_D3(d7, r8[c], V14[c], V15[c], V16);
#define GX_D9(p) GX_D3(p, fma(p##13, kn[c], GX_D8(p, k1[c], k6[c], k7[c], k8[c], k9[c], k10[c], k11[c], k12[c])), k14[c], k15[c], k16[c])
                    const double v5 = GX_D9(d4), v6 = GX_D9(d5), v7 = GX_D9(d6), v8 = GX_D9(d7);
#undef GX_D9
#undef GX_D3
                    const double xd = xn[c] - x[c], xb = fma(h, v[c], -xd), x4 = fma(-h, vn[c], xd) - xb;
                    const double vd = vn[c] - v[c], vb = fma(h, k1[c], -vd), v4 = fma(-h, kn[c], vd) - vb;
                    double *o = out + c * rows + i0 + j;
                    int64_t slot = out_slot;
                    for (next = kept; next < out_end; next += A.out_stride, slot++) {
                        const double s = ddiv(t[next] - xold, hout);
                        const double s1 = 1.0 - s;
                        if (active) {
                            __stcs(o + slot * n, fma(s, fma(s1, fma(s, fma(s1, fma(s, fma(s1, fma(s, x8, x7), x6), x5), x4),
                                                               xb), xd), x[c]));
                            __stcs(o + 3 * rows + slot * n,
                                   fma(s, fma(s1, fma(s, fma(s1, fma(s, fma(s1, fma(s, v8, v7), v6), v5), v4), vb), vd), v[c]));
                        }
                    }
                    if (c == 2) out_slot = slot;
                }
                kept = next;
#undef GX_D8
            }
            out_idx = out_end;

            for (int c = 0; c < 3; c++) {
                k1[c] = kn[c];
                x[c] = xn[c];
                v[c] = vn[c];
            }
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
    if (G > 1) cluster_sync_all();  // no CTA leaves while another may still write to it

    if (!A.save_all && active)
        for (int c = 0; c < 3; c++) {
            out[c * n + i0 + j] = x[c];
            out[(3 + c) * n + i0 + j] = v[c];
        }
    if (j == 0) {
        status[b] = idid;
        if (stats) {
            stats[4 * b + 0] = nfcn;
            stats[4 * b + 1] = nstep;
            stats[4 * b + 2] = naccpt;
            stats[4 * b + 3] = nrejct;
        }
    }
}
#undef ACC

// One cluster of one-warp CTAs per batch.
static cudaError_t launch_static(const DevPot &dp, const DopArgs &A, int G, const double *w0, int64_t n, const double *t,
                                 double *out, int32_t *status, int64_t *stats, cudaStream_t st) {
    const int64_t nbatches = (n + A.nbatch - 1) / A.nbatch;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(nbatches * G));
    cfg.blockDim = dim3(32);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = G;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return dp.has_scf ? cudaLaunchKernelEx(&cfg, dop853_static_kernel<true>, dp, A, G, w0, n, t, out, status, stats)
                      : cudaLaunchKernelEx(&cfg, dop853_static_kernel<false>, dp, A, G, w0, n, t, out, status, stats);
}

// The kernel that takes a call.
static int dop853_form(const DevPot &dp, const DevFrame &df, const DopArgs &A, int64_t n) {
    // Few orbits: one coordinate per lane.
    if (dop853_axis_takes(dp, df, A, n)) return GX_DOP853_AXIS;
    // A static frame and a batch that fills one to eight warps (the portable cluster
    // size): a cluster per batch.  Several batches of at most 16 orbits stay with the general
    // kernel, where two of them share a warp and with it each FP64 instruction.
    const int64_t nbatches = (n + A.nbatch - 1) / A.nbatch;
    const int64_t G = ((A.nbatch < n ? A.nbatch : n) + 31) / 32;
    if (df.type == GX_FRAME_STATIC && G <= NYS_MAX_WARPS && (A.nbatch > 16 || nbatches == 1) && nbatches * G < ((int64_t)1 << 31))
        return GX_DOP853_CLUSTER;
    return GX_DOP853_GENERAL;
}

}  // namespace gx

extern "C" int gx_dop853_form(const gx_potential *pot, const gx_frame *frame, int64_t n, int32_t nbatch, int32_t *form) {
    gx::DevPot dp;
    gx::DevFrame df;
    int rc = gx::pack_potential(pot, &dp);
    if (rc) return rc;
    rc = gx::pack_frame(frame, &df);
    if (rc) return rc;
    GX_CHECK_ARG(n >= 0, "n < 0");
    GX_CHECK_ARG(nbatch >= 1 && nbatch <= 1024, "nbatch must be in [1, 1024] (got %d)", nbatch);
    GX_CHECK_ARG(form, "NULL pointer");
    gx::DopArgs A = {};
    A.nbatch = nbatch;
    *form = gx::dop853_form(dp, df, A, n);
    return GX_OK;
}

extern "C" int gx_dop853_integrate_hamiltonian(const gx_potential *pot, const gx_frame *frame, const double *w0,
                                               int64_t n, const double *t, int64_t ntimes, double atol,
                                               double rtol, int64_t nmax, double dt_max, int64_t nstiff,
                                               int32_t save_all, int32_t nbatch, int64_t out_stride,
                                               double *w_out, int32_t *status, int64_t *stats, void *stream) {
    gx::DevPot dp;
    gx::DevFrame df;
    int rc = gx::pack_potential(pot, &dp);
    if (rc) return rc;
    rc = gx::pack_frame(frame, &df);
    if (rc) return rc;
    GX_CHECK_ARG(n >= 0, "n < 0");
    GX_CHECK_ARG(ntimes >= 2, "ntimes must be >= 2 (got %lld)", (long long)ntimes);
    GX_CHECK_ARG(nbatch >= 1 && nbatch <= 1024, "nbatch must be in [1, 1024] (got %d)", nbatch);
    GX_CHECK_ARG(out_stride >= 1, "out_stride must be >= 1");
    GX_CHECK_ARG(nmax >= 0, "nmax must be >= 0 (0 = gala's default 1e6)");
    GX_CHECK_ARG(atol >= 0 && rtol >= 0, "tolerances must be non-negative");
    if (n == 0) return GX_OK;
    GX_CHECK_ARG(w0 && t && w_out && status, "NULL array");
    gx::DopArgs A;
    memset(&A, 0, sizeof(A));
    A.cancel = gx::cancel_flag();
    A.atol = atol;
    A.rtol = rtol;
    A.dt_max = dt_max;
    A.nmax = nmax;
    A.nstiff = nstiff;
    A.ntimes = ntimes;
    A.out_stride = out_stride;
    A.n_out = (ntimes - 1) / out_stride + 1;
    A.save_all = save_all ? 1 : 0;
    A.nbatch = nbatch;
    const int64_t nbatches = (n + nbatch - 1) / nbatch;
    cudaStream_t st = gx::as_stream(stream);
    const int form = gx::dop853_form(dp, df, A, n);
    if (form == GX_DOP853_AXIS) return gx::launch_dop853_axis(dp, df, A, w0, n, t, w_out, status, stats, st);
    if (form == GX_DOP853_CLUSTER) {
        const int G = (int)(((nbatch < n ? nbatch : n) + 31) / 32);
        const cudaError_t e = gx::launch_static(dp, A, G, w0, n, t, w_out, status, stats, st);
        if (e != cudaSuccess) {
            gx::set_error("dop853 launch failed: %s", cudaGetErrorString(e));
            return GX_ERR_CUDA;
        }
        return gx::check_launch("dop853");
    }
    // Two batches share a CTA when that fills the warps better (a 100-orbit batch
    // alone leaves 28 lanes of its fourth warp idle, and the FP64 pipe costs a
    // warp instruction whatever its mask); they step in lock-step.
    const int t1 = ((nbatch + 31) / 32) * 32, t2 = ((2 * nbatch + 31) / 32) * 32;
    const bool pair = !dp.has_scf && t2 <= 256 && t2 < 2 * t1;
    const int threads = pair ? t2 : t1;
    const unsigned grid = (unsigned)(pair ? (nbatches + 1) / 2 : nbatches);
    if (pair)
        gx::dop853_kernel<256, false, 2><<<grid, threads, 0, st>>>(dp, df, A, w0, n, t, w_out, status, stats);
    else if (threads <= 256 && !dp.has_scf)
        gx::dop853_kernel<256, false, 1><<<grid, threads, 0, st>>>(dp, df, A, w0, n, t, w_out, status, stats);
    else if (threads <= 256)
        gx::dop853_kernel<256, true, 1><<<grid, threads, 0, st>>>(dp, df, A, w0, n, t, w_out, status, stats);
    else if (!dp.has_scf)
        gx::dop853_kernel<1024, false, 1><<<grid, threads, 0, st>>>(dp, df, A, w0, n, t, w_out, status, stats);
    else
        gx::dop853_kernel<1024, true, 1><<<grid, threads, 0, st>>>(dp, df, A, w0, n, t, w_out, status, stats);
    return gx::check_launch("dop853");
}

namespace gx {
__global__ void selfcheck_fast64_kernel(const double *__restrict__ x, int64_t n, double *__restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double v = x[i];
    out[i] = fast::log_f(v);
    out[n + i] = log(v);
    out[2 * n + i] = fast::sqrt_f(v);
    out[3 * n + i] = fast::rcp_f(v);
}
}  // namespace gx

extern "C" int gx_selfcheck_fast64(const double *x, int64_t n, double *out, void *stream) {
    GX_CHECK_ARG(n >= 0, "n < 0");
    if (n == 0) return GX_OK;
    GX_CHECK_ARG(x && out, "NULL array");
    gx::selfcheck_fast64_kernel<<<(unsigned)((n + 255) / 256), 256, 0, gx::as_stream(stream)>>>(x, n, out);
    return gx::check_launch("selfcheck_fast64");
}

namespace gx {
__global__ void selfcheck_ipipe_kernel(const double *__restrict__ x, const double *__restrict__ y, int64_t n,
                                       double *__restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double rs;
    out[i] = ip::sqrt_rn(x[i]);
    out[n + i] = ip::div_rn(x[i], y[i]);
    out[2 * n + i] = sqrt(x[i]);
    out[3 * n + i] = x[i] / y[i];
    out[4 * n + i] = ip::sqrt_rsqrt_n(x[i], rs);
    out[5 * n + i] = rs;
}
}  // namespace gx

extern "C" int gx_selfcheck_ipipe(const double *x, const double *y, int64_t n, double *out, void *stream) {
    GX_CHECK_ARG(n >= 0, "n < 0");
    if (n == 0) return GX_OK;
    GX_CHECK_ARG(x && y && out, "NULL array");
    gx::selfcheck_ipipe_kernel<<<(unsigned)((n + 255) / 256), 256, 0, gx::as_stream(stream)>>>(x, y, n, out);
    return gx::check_launch("selfcheck_ipipe");
}
