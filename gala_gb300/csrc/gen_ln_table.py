"""Generate gx_ln_table.cuh: the table of the fixed-point logarithm in
gx_ipipe.cuh (ln x = k ln 2 - ln c_j + ln(1 + r), r = m c_j - 1).

For j = 0..511, c_j is 1 / (1 + (j + 1/2) / 512) rounded to 32 fraction bits (so
|r| < 2^-9.9 for m in [1 + j / 512, 1 + (j + 1) / 512)) and T_j = -ln(c_j) of the
rounded c_j, rounded to 64 fraction bits, from 60-digit arithmetic.  Run:
    python gen_ln_table.py > gx_ln_table.cuh
"""
import mpmath

mpmath.mp.dps = 60


def main():
    out = ["// gx_ln_table.cuh -- generated by gen_ln_table.py; do not edit.",
           "// Table of the fixed-point logarithm (gx_ipipe.cuh): for j = 0..511",
           "// {T_j low word, T_j high word, c_j 2^32, 0}, c_j ~ 1 / (1 + (j + 1/2) / 512), T_j = -ln(c_j) 2^64.",
           "#pragma once", "", "#include <cstdint>", "", "namespace gx {", "namespace ip {", "",
           "#ifdef __CUDACC__", "static __device__ const __align__(16)", "#else", "static const", "#endif",
           "uint32_t LN_TAB[512][4] = {"]
    for j in range(512):
        c = int(mpmath.nint(2 ** 32 / (1 + (mpmath.mpf(j) + mpmath.mpf(1) / 2) / 512)))
        t = int(mpmath.nint(-mpmath.log(mpmath.mpf(c) / 2 ** 32) * 2 ** 64))
        out.append(f"    {{0x{t & 0xffffffff:08x}u, 0x{t >> 32:08x}u, 0x{c:08x}u, 0u}},")
    out += ["};", "", f"constexpr uint64_t LN2_64 = 0x{int(mpmath.nint(mpmath.log(2) * 2 ** 64)):016x}ull;  // ln 2 at 2^-64",
            "", "}  // namespace ip", "}  // namespace gx", ""]
    print("\n".join(out))


if __name__ == "__main__":
    main()
