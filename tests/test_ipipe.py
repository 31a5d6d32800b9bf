"""CPU check of the fixed-point cores of gala_gb300/csrc/gx_ipipe.cuh (plain
integer C++, compiled here with the host compiler): with FP32 seeds off by up to
4 units in the last place, the square root and the quotient have the bits of IEEE
arithmetic, the reciprocal is within one unit, and the logarithm within 0.85 ulp
(half an ulp of rounding, 3 units of 2^-64 of summation and 2^-61 of the series'
32-bit coefficients against results of at least 2^-6, whose ulp is 2^-59)."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "gala_gb300" / "csrc"

SRC = r"""
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include "gx_ipipe.cuh"
using namespace gx::ip;
static uint64_t bits(double x) { uint64_t b; memcpy(&b, &x, 8); return b; }
static double dbl(uint64_t b) { double x; memcpy(&x, &b, 8); return x; }
static uint32_t fbits(float x) { uint32_t b; memcpy(&b, &x, 4); return b; }
static float flt(uint32_t b) { float x; memcpy(&x, &b, 4); return x; }
static uint32_t top(uint64_t f) { return (uint32_t)(f >> 29); }
int main(int argc, char **argv) {
    const long n = atol(argv[1]);
    const int mode = atoi(argv[2]);  // where the 52-bit fractions lie
    std::mt19937_64 g(mode + 1);
    const uint64_t F = (1ull << 52) - 1;
    auto frac = [&]() -> uint64_t {
        uint64_t f = g() & F;
        if (mode == 1) f = g() % 64;                       // just above a power of two
        if (mode == 2) f = F - g() % 64;                   // just below
        if (mode == 3) f &= ~((1ull << (g() % 52)) - 1);   // few significant bits
        if (mode == 4) { const double s = (double)((1ull << 26) + (g() & 0x3ffffff)); f = bits(s * s + (double)(int)(g() % 3) - 1) & F; }  // squares
        if (mode == 5) f = ((g() % 512) << 43) + (g() % 64) - 32 & F;  // edges of the table's intervals
        return f;
    };
    long bad_div = 0, bad_rcp = 0, bad_sqrt = 0;
    double ln = 0;
    for (long i = 0; i < n; i++) {
        const uint64_t fa = frac(), fb = i % 3 ? frac() : g() & F;
        const double a = dbl((1023ull << 52) | fa), b = dbl((1023ull << 52) | fb);
        const int off = (int)(g() % 9) - 4;
        const uint64_t mb = ((1ull << 52) | fb) << 11;
        const uint64_t y = rcp63((uint32_t)(mb >> 32), (uint32_t)mb, seed24(fbits(1.0f / flt(0x3f800000u | top(fb))) + off));
        if (std::fabs((double)((y + 512) >> 10) * 0x1p-53 - 1.0 / b) > 0x1p-53) bad_rcp++;
        uint64_t A = (1ull << 52) | fa;
        const uint64_t B = (1ull << 52) | fb;
        const int less = A < B;
        if ((double)div53_rn(A << less, B, y) * 0x1p-52 != std::ldexp(a, less) / b) bad_div++;
        for (int odd = 0; odd < 2; odd++) {
            const uint64_t M = ((1ull << 52) | fa) << 11, v = odd ? M : M >> 1;
            const uint64_t r = rsqrt63(v, seed24(fbits(1.0f / std::sqrt(flt(((127u + odd) << 23) | top(fa)))) + off));
            if ((double)sqrt53_rn(v, r) * 0x1p-52 != std::sqrt(std::ldexp(a, odd))) bad_sqrt++;
        }
        const uint32_t k = i % 2 ? (uint32_t)(g() % 1024) : 0;
        const double x = dbl(((uint64_t)(1023 + k) << 52) | fa);
        if (x < 1 + 0x1p-6) continue;
        const uint32_t *e = LN_TAB[(bits(x) >> 43) & 511];
        const uint64_t M = ((1ull << 52) | fa) << 11;
        int s;
        const uint64_t R = ln_sum53(k, ln64((uint32_t)(M >> 32), (uint32_t)M, e[2], ((uint64_t)e[1] << 32) | e[0]), s);
        const long double ref = logl((long double)x);
        const double err = (double)fabsl((ldexpl((long double)R, s - 53) - ref) / ldexpl(1, ilogbl(ref) - 52));
        ln = err > ln ? err : ln;
    }
    printf("%ld %ld %ld %.6f\n", bad_div, bad_rcp, bad_sqrt, ln);
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    d = tmp_path_factory.mktemp("ipipe")
    (d / "h.cpp").write_text(SRC)
    subprocess.run([cxx, "-O2", "-std=c++17", f"-I{CSRC}", str(d / "h.cpp"), "-o", str(d / "h")], check=True)
    return d / "h"


@pytest.mark.parametrize("mode", range(6))
def test_cores(harness, mode):
    out = subprocess.run([str(harness), "400000", str(mode)], capture_output=True, text=True, check=True).stdout.split()
    assert out[:3] == ["0", "0", "0"], out
    assert float(out[3]) <= 0.85
