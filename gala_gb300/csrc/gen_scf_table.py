"""Generate gx_scf_table.cuh: the constants of the SCF recurrences in gx_scf.cuh,
for l = 0..15 and n = 0..23, from 60-digit arithmetic.  With a = 2 l + 3/2:

    GEG1[l][n] = 2 (n + a - 1) / n,  GEG2[l][n] = (n + 2 a - 2) / n
        C_n^a(x) = GEG1 x C_{n-1}^a - GEG2 C_{n-2}^a         (n >= 1)
    GEGD[l][n] = (n + a) / a
        C_n^{a+1} = C_{n-2}^{a+1} + GEGD C_n^a
    YNORM[l][m] = sqrt((2 l + 1) (l - m)! / (l + m)!)
    INT[k] = k, INV[k] = 1 / k
Run:
    python gen_scf_table.py > gx_scf_table.cuh
"""
import mpmath

mpmath.mp.dps = 60
NL, NN = 16, 24


def rows(name, dims, f):
    out = [f"static __constant__ double {name}{dims} = {{"]
    for l in range(NL):
        out.append("    {" + ", ".join(float(x).hex() for x in f(l)) + "},")
    return out + ["};"]


def main():
    M = mpmath.mpf
    a = lambda l: 2 * M(l) + M(3) / 2  # noqa: E731
    out = ["// gx_scf_table.cuh -- generated by gen_scf_table.py; do not edit.",
           "// Constants of the Gegenbauer, Legendre and normalisation recurrences of gx_scf.cuh.",
           "#pragma once", "", "namespace gx {", "namespace scf {", ""]
    out += rows("GEG1", f"[{NL}][{NN}]", lambda l: [0 if n == 0 else 2 * (n + a(l) - 1) / n for n in range(NN)])
    out += rows("GEG2", f"[{NL}][{NN}]", lambda l: [0 if n == 0 else (n + 2 * a(l) - 2) / n for n in range(NN)])
    out += rows("GEGD", f"[{NL}][{NN}]", lambda l: [(n + a(l)) / a(l) for n in range(NN)])
    out += rows("YNORM", f"[{NL}][{NL}]", lambda l: [mpmath.sqrt((2 * l + 1) * mpmath.factorial(l - m) / mpmath.factorial(l + m))
                                                     if m <= l else 0 for m in range(NL)])
    out += [f"static __constant__ double INT[{2 * NL}] = {{" + ", ".join(float(k).hex() for k in range(2 * NL)) + "};",
            f"static __constant__ double INV[{NL}] = {{" + ", ".join(float(M(1) / k if k else 0).hex() for k in range(NL)) + "};",
            "", "}  // namespace scf", "}  // namespace gx", ""]
    print("\n".join(out))


if __name__ == "__main__":
    main()
