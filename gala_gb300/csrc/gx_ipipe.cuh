// gx_ipipe.cuh -- FP64 square root, reciprocal, quotient and logarithm in 64-bit
// fixed point, on the integer pipe.
//
// The FP64 unit of this part is shared by the four sub-partitions of an SM and
// takes one warp instruction per 19 cycles (76 per sub-partition; measured, and
// the same for 1 or 32 active lanes), while a 32 x 32 -> 64-bit multiply-add
// costs 5 cycles of a sub-partition and an integer add or shift about 1.5.  The
// library's sqrt and a / b are 8 FP64 instructions (608 cycles), 1/x 5, log ~30.
// The same functions as fixed-point Newton steps are 60 to 130 cycles of integer
// work that runs beside the FP64 unit instead of on it.
//
// Method, all from the mathematics:
//   1/m, m in [1, 2)       FP32 seed y0 (relative error < 2^-21), d = m y0 - 1 exactly,
//                          y = y0 (1 - d + d^2); the error d^3 is below 2^-63
//   1/sqrt(v), v in [1, 4) FP32 seed, d = v y0^2 - 1, y = y0 (1 - d/2 + 3/8 d^2)
//   sqrt, a / b            the 62-bit approximation rounded to 53 bits, then the
//                          sign of the exact remainder (mod 2^64, which holds it)
//                          moves it by one unit where the rounding was wrong:
//                          correctly rounded, the bits of IEEE sqrt and division
//   ln x                   x = 2^k m, r = m c_j - 1 (c_j ~ 1/m from a 512-entry
//                          table, exact in 96 bits, |r| < 2^-9.9),
//                          ln x = k ln 2 - ln c_j + r - r^2 (1/2 - r (1/3 - ...))
// Arguments or results outside the normal range (and ln near or below 1, where
// a fixed-point sum loses relative accuracy) go to the library functions.
//
// The fixed-point cores are plain integer C++ (host and device), so they are
// checked on the CPU against IEEE sqrt and division with perturbed seeds
// (tests/test_ipipe.py) and on the GPU against the library (gx_selfcheck_ipipe).
#pragma once

#include <cstdint>

#include "gx_ln_table.cuh"

#ifdef __CUDACC__
#define GX_HD __host__ __device__ __forceinline__
#else
#define GX_HD inline
#endif

namespace gx {
namespace ip {

// ---- cores -----------------------------------------------------------------

GX_HD int clz32(uint32_t x) {
#ifdef __CUDA_ARCH__
    return __clz((int)x);
#else
    return __builtin_clz(x);
#endif
}
GX_HD int clz64(uint64_t x) {
#ifdef __CUDA_ARCH__
    return __clzll((long long)x);
#else
    return __builtin_clzll(x);
#endif
}

// High 64 bits of a b, low by at most 2 units (the low halves' product and
// two carries are not formed).
GX_HD uint64_t mulhi_a(uint64_t a, uint64_t b) {
    const uint32_t a0 = (uint32_t)a, a1 = (uint32_t)(a >> 32), b0 = (uint32_t)b, b1 = (uint32_t)(b >> 32);
    return (uint64_t)a1 * b1 + (((uint64_t)a1 * b0) >> 32) + (((uint64_t)a0 * b1) >> 32);
}

// FP32 seed in [0.5, 1) as a 24-bit integer, scale 2^-24 (a seed that the
// approximate instruction put just outside is clamped).
GX_HD uint32_t seed24(uint32_t fbits) {
    fbits = fbits < 0x3f000000u ? 0x3f000000u : fbits;
    fbits = fbits > 0x3f7fffffu ? 0x3f7fffffu : fbits;
    return (fbits & 0x7fffffu) | 0x800000u;
}

// 1/m, m in [1, 2) at scale 2^-63 (mh, ml), Y the 24-bit seed: (0.5, 1] at scale 2^-63.
GX_HD uint64_t rcp63(uint32_t mh, uint32_t ml, uint32_t Y) {
    const uint64_t p = (uint64_t)ml * Y;
    const uint64_t P = (uint64_t)mh * Y + (p >> 32);                       // m y0 at 2^-55
    const int64_t d = (int64_t)(((P - (1ull << 55)) << 28) | ((uint32_t)p >> 4));  // m y0 - 1 at 2^-83
    const int32_t dh = (int32_t)(d >> 32);
    const int64_t g = d - (((int64_t)dh * dh) >> 19);                      // d - d^2
    const int64_t c = (int64_t)(int32_t)Y * (int32_t)(g >> 32) + (int64_t)(((uint64_t)Y * (uint32_t)g) >> 32);
    return ((uint64_t)Y << 39) - (uint64_t)(c >> 12);                      // c at 2^-75
}

// 1/sqrt(v), v in [1, 4) at scale 2^-62, Y the 24-bit seed: (0.5, 1] at scale 2^-63.
GX_HD uint64_t rsqrt63(uint64_t v, uint32_t Y) {
    const uint32_t vh = (uint32_t)(v >> 32), vl = (uint32_t)v;
    const uint64_t Y2 = (uint64_t)Y * Y;  // scale 2^-48
    const uint32_t yh = (uint32_t)(Y2 >> 32), yl = (uint32_t)Y2;
    // v y0^2 - 1 at 2^-78: the 1 is 2^78, a multiple of 2^64
    const int64_t d = (int64_t)((uint64_t)vh * yl + (uint64_t)vl * yh + (((uint64_t)vl * yl) >> 32) +
                                ((uint64_t)(uint32_t)(vh * yh) << 32));
    const int32_t dh = (int32_t)(d >> 32);
    const int64_t g = (d >> 1) - (((int64_t)dh * (3 * dh)) >> 17);         // d/2 - 3/8 d^2
    const int64_t c = (int64_t)(int32_t)Y * (int32_t)(g >> 32) + (int64_t)(((uint64_t)Y * (uint32_t)g) >> 32);
    return ((uint64_t)Y << 39) - (uint64_t)(c >> 7);                       // c at 2^-70
}

// sqrt(v) rounded to 53 bits ([2^52, 2^53]) from y = 1/sqrt(v): within 0.51 units.
GX_HD uint64_t sqrt53(uint64_t v, uint64_t y) { return (mulhi_a(v, y) + 256) >> 9; }

// The same, correctly rounded: D = v 2^42 - R^2 decides (all integers; sqrt(X)
// rounds to R exactly where -R < X - R^2 <= R).
GX_HD uint64_t sqrt53_rn(uint64_t v, uint64_t y) {
    const uint64_t R = sqrt53(v, y);
    const int64_t D = (int64_t)((v << 42) - R * R);
    return R + (uint64_t)(D > (int64_t)R) - (uint64_t)(D <= -(int64_t)R);
}

// a / b in [1, 2) for 53-bit integers with b <= a < 2 b, y = 1/b as from rcp63
// (b taken as b 2^-52): correctly rounded to 53 bits ([2^52, 2^53]).
GX_HD uint64_t div53_rn(uint64_t a, uint64_t b, uint64_t y) {
    const uint64_t q = (mulhi_a(a << 10, y) + 256) >> 9;  // (a 2^10)(y) >> 64 at 2^-61
    const int64_t r2 = (int64_t)((a << 53) - 2 * (q * b));  // twice the remainder
    return q + (uint64_t)(r2 > (int64_t)b) - (uint64_t)(r2 < -(int64_t)b);
}

// ln m at scale 2^-64 for m in [1, 2) at scale 2^-63, c = c_j at scale 2^-32 and
// T = -ln c_j at scale 2^-64 (LN_TAB); within 3 units, so near m = 1 it may wrap
// just below zero.
GX_HD uint64_t ln64(uint32_t mh, uint32_t ml, uint32_t c, uint64_t T) {
    const uint64_t p = (uint64_t)ml * c;
    const uint64_t P = (uint64_t)mh * c + (p >> 32);                                 // m c at 2^-63
    const int64_t r = (int64_t)(((P - (1ull << 63)) << 9) | ((uint32_t)p >> 23));    // r at 2^-72
    // r = rh 2^32 + rl with rl signed, so that rh^2 + 2 rh rl never falls below zero
    const int32_t rl = (int32_t)(uint32_t)r;
    const int32_t rh = (int32_t)(r >> 32) + (int32_t)((uint32_t)r >> 31);            // 2^-40
    const uint64_t r2 = (uint64_t)((int64_t)rh * rh + (((int64_t)rh * rl) >> 31));   // r^2 at 2^-80
    // w = 1/3 - r (1/4 - r (1/5 - r/6)) at 2^-32, in 8-bit steps of the scale
    int32_t w = 43;
    w = 13107 - (int32_t)(((int64_t)rh * w) >> 32);
    w = 4194304 - (int32_t)(((int64_t)rh * w) >> 32);
    w = 1431655765 - (int32_t)(((int64_t)rh * w) >> 32);
    const uint64_t q = (1ull << 63) - (uint64_t)(((int64_t)rh * w) >> 8);            // 1/2 - r w at 2^-64
    const int64_t l1p = r - (int64_t)(mulhi_a(r2, q) >> 8);                          // ln(1 + r) at 2^-72
    return T + (uint64_t)(l1p >> 8);
}

// k ln 2 + F rounded to 53 bits: R 2^-53 2^s with R in [2^52, 2^53] (F as from
// ln64; k > 0 or F well above 0).
GX_HD uint64_t ln_sum53(uint32_t k, uint64_t F, int &s) {
    const uint64_t u = (uint64_t)k * (uint32_t)LN2_64, u2 = (uint64_t)k * (uint32_t)(LN2_64 >> 32) + (u >> 32);
    const uint64_t b = k ? 8u : 0u;  // keeps F + b above zero where F wrapped
    const uint64_t f = ((u2 << 32) | (uint32_t)u) - b;
    F += b;
    F += f;
    const uint32_t ip = (uint32_t)(u2 >> 32) + (F < f ? 1u : 0u);
    // normalised: top bit 63, value V 2^-64 2^s (both forms, one of them taken: a
    // branch here would part the lanes of a warp)
    const int up = 32 - clz32(ip | 1u), down = clz64(F | 1u);
    const uint64_t Vu = ((uint64_t)ip << (64 - up)) | (F >> up), Vd = F << down;
    const uint64_t V = ip ? Vu : Vd;
    s = ip ? up : -down;
    return (V >> 11) + ((V >> 10) & 1u);
}

// ---- pieces of a double ------------------------------------------------------

struct Mant {
    uint32_t hi, lo;  // 1.f at scale 2^-63
};
GX_HD Mant mant63(uint32_t hi, uint32_t lo) {
    return {0x80000000u | (hi << 11) | (lo >> 21), lo << 11};
}

#ifdef __CUDACC__

__device__ __forceinline__ uint32_t rcp_seed(uint32_t fb) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(fb)));
    return seed24(__float_as_uint(y));
}
__device__ __forceinline__ uint32_t rsqrt_seed(uint32_t fb) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(fb)));
    return seed24(__float_as_uint(y));
}
// top 23 mantissa bits of a double
__device__ __forceinline__ uint32_t top23(uint32_t hi, uint32_t lo) { return ((hi << 3) | (lo >> 29)) & 0x7fffffu; }
// normal and not negative
__device__ __forceinline__ bool normal_pos(uint32_t hi) { return hi - 0x00100000u < 0x7fe00000u; }
// |x| in [2^-511, 2^511): quotients of two such numbers are normal
__device__ __forceinline__ bool mid_range(uint32_t hi) { return (hi & 0x7fffffffu) - (512u << 20) < (1022u << 20); }
// (e + 1) 2^52 + R with R in [2^52, 2^53]: the double of value R 2^-52 2^e, ebits = (e + 1022) << 20
__device__ __forceinline__ double pack53(uint64_t R, uint32_t ebits) {
    return __longlong_as_double((long long)(R + ((uint64_t)ebits << 32)));
}

// v in [1, 4) at 2^-62 and the FP32 argument of the seed, x = v 4^h; hbits = (h + 1022) << 20
struct SqrtArg {
    uint64_t v;
    uint32_t fb, hbits;
};
__device__ __forceinline__ SqrtArg sqrt_arg(uint32_t hi, uint32_t lo) {
    const Mant m = mant63(hi, lo);
    const uint64_t M = ((uint64_t)m.hi << 32) | m.lo;
    const uint32_t odd = ((hi >> 20) & 1u) ^ 1u;  // biased 1023 is an even exponent
    SqrtArg a;
    a.v = M >> (1u - odd);
    a.fb = ((127u + odd) << 23) | top23(hi, lo);
    a.hbits = ((((hi >> 20) - odd + 1023u) >> 1) - 1u) << 20;  // (k' / 2 + 1022), k' = k - odd
    return a;
}

// The forms named _u take any bits and are right where ok_ says so; a straight
// run of them leaves the compiler free to interleave their dependent chains (190
// to 430 cycles each alone), which a branch in each would forbid.

// IEEE sqrt.
__device__ __forceinline__ bool ok_sqrt(double x) { return normal_pos((uint32_t)__double2hiint(x)); }
__device__ __forceinline__ double sqrt_rn_u(double x) {
    const SqrtArg a = sqrt_arg((uint32_t)__double2hiint(x), (uint32_t)__double2loint(x));
    return pack53(sqrt53_rn(a.v, rsqrt63(a.v, rsqrt_seed(a.fb))), a.hbits);
}
__device__ __forceinline__ double sqrt_rn(double x) { return ok_sqrt(x) ? sqrt_rn_u(x) : sqrt(x); }
// sqrt within 0.51 ulp.
__device__ __forceinline__ double sqrt_n(double x) {
    const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
    if (!normal_pos(hi)) return sqrt(x);
    const SqrtArg a = sqrt_arg(hi, lo);
    return pack53(sqrt53(a.v, rsqrt63(a.v, rsqrt_seed(a.fb))), a.hbits);
}
// sqrt(x) (returned) and 1 / sqrt(x), each within 0.51 ulp, from one core.
__device__ __forceinline__ double sqrt_rsqrt_u(double x, double &rs) {
    const SqrtArg a = sqrt_arg((uint32_t)__double2hiint(x), (uint32_t)__double2loint(x));
    const uint64_t y = rsqrt63(a.v, rsqrt_seed(a.fb));
    // 1 / sqrt(x) = y 2^-h, y in (0.5, 1] at 2^-63: R = y 2^53 in [2^52, 2^53], exponent -h - 1
    rs = pack53((y + 512) >> 10, (2u * 1022u - 1u) * (1u << 20) - a.hbits);
    return pack53(sqrt53(a.v, y), a.hbits);
}
__device__ __forceinline__ double rsqrt_u(double x) {
    double rs;
    sqrt_rsqrt_u(x, rs);
    return rs;
}
__device__ __forceinline__ double sqrt_rsqrt_n(double x, double &rs) {
    if (ok_sqrt(x)) return sqrt_rsqrt_u(x, rs);
    const double s = sqrt(x);
    rs = 1.0 / s;
    return s;
}
// 1/x within 0.51 ulp.
__device__ __forceinline__ bool ok_rcp(double x) { return mid_range((uint32_t)__double2hiint(x)); }
__device__ __forceinline__ double rcp_u(double x) {
    const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
    const Mant m = mant63(hi, lo);
    const uint64_t y = rcp63(m.hi, m.lo, rcp_seed(0x3f800000u | top23(hi, lo)));
    const uint32_t eb = (2044u << 20) - (hi & 0x7ff00000u);  // -k - 1 + 1022
    return pack53((y + 512) >> 10, eb | (hi & 0x80000000u));
}
__device__ __forceinline__ double rcp_n(double x) { return ok_rcp(x) ? rcp_u(x) : 1.0 / x; }
// IEEE a / b.
__device__ __forceinline__ double div_rn_u(double a, double b) {
    const uint32_t ah = (uint32_t)__double2hiint(a), al = (uint32_t)__double2loint(a);
    const uint32_t bh = (uint32_t)__double2hiint(b), bl = (uint32_t)__double2loint(b);
    const Mant m = mant63(bh, bl);
    const uint64_t y = rcp63(m.hi, m.lo, rcp_seed(0x3f800000u | top23(bh, bl)));
    uint64_t A = ((uint64_t)(0x00100000u | (ah & 0xfffffu)) << 32) | al;
    const uint64_t B = ((uint64_t)(0x00100000u | (bh & 0xfffffu)) << 32) | bl;
    const uint32_t less = A < B;
    A <<= less;
    const uint64_t q = div53_rn(A, B, y);
    const uint32_t eb = (ah & 0x7ff00000u) - (bh & 0x7ff00000u) + ((1022u - less) << 20);
    return __longlong_as_double((long long)((q + ((uint64_t)eb << 32)) ^ ((uint64_t)((ah ^ bh) & 0x80000000u) << 32)));
}
__device__ __forceinline__ bool ok_div(double a, double b) { return ok_rcp(a) & ok_rcp(b); }
__device__ __forceinline__ double div_rn(double a, double b) { return ok_div(a, b) ? div_rn_u(a, b) : a / b; }
// Whether ln_n takes x: finite and at least 1 + 2^-6.
__device__ __forceinline__ bool ln_range(double x) {
    return (uint32_t)__double2hiint(x) - 0x3ff04000u < 0x7ff00000u - 0x3ff04000u;
}
// ln x within 0.65 ulp, x in ln_range.
__device__ __forceinline__ double ln_n(double x) {
    const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
    const uint4 e = __ldg(reinterpret_cast<const uint4 *>(LN_TAB) + ((hi >> 11) & 511u));  // {-ln c lo, hi, c, 0}
    const Mant m = mant63(hi, lo);
    uint64_t F = ln64(m.hi, m.lo, e.z, ((uint64_t)e.y << 32) | e.x);
    int s;
    const uint64_t R = ln_sum53((hi >> 20) - 1023u, F, s);
    return pack53(R, (uint32_t)(s + 1021) << 20);
}

#endif  // __CUDACC__

}  // namespace ip
}  // namespace gx
