"""Generate gx_dop853_nystrom.cuh: the DOP853 tableau (gx_dop853_tableau.cuh) in
the form it takes for x' = v, v' = a(x) (a static frame): the position of a
stage needs only the accelerations,

    x_i = x + h c_i v + h^2 sum_l (A^2)_il a_l,   x_new = x + h v + h^2 sum_l (b A)_l a_l,

and so do the error estimates of the positions, with (er A) and ((b - bhh) A).
Products in 40-digit arithmetic, rounded once.  Run:
    python gen_dop853_nystrom.py > gx_dop853_nystrom.cuh
"""
import re
from pathlib import Path

import mpmath

mpmath.mp.dps = 40


def main():
    text = (Path(__file__).resolve().parent / "gx_dop853_tableau.cuh").read_text()
    T = {m.group(1): mpmath.mpf(m.group(2)) for m in re.finditer(r"constexpr double (\w+) = ([-0-9.Ee+]+);", text)}
    A = mpmath.matrix(13, 13)
    for i in range(2, 13):
        for j in range(1, i):
            A[i, j] = T.get(f"a{i}{j}", mpmath.mpf(0))
    b, er = mpmath.matrix(1, 13), mpmath.matrix(1, 13)
    for j in range(1, 13):
        b[0, j], er[0, j] = T.get(f"b{j}", mpmath.mpf(0)), T.get(f"er{j}", mpmath.mpf(0))
    bhh = b.copy()
    for j, k in ((1, 1), (9, 2), (12, 3)):
        bhh[0, j] -= T[f"bhh{k}"]
    out = ["// gx_dop853_nystrom.cuh -- generated by gen_dop853_nystrom.py; do not edit.",
           "// DOP853 for x' = v, v' = a(x): nIJ = (A^2)_IJ, nbJ = (b A)_J, nerJ = (er A)_J,",
           "// nbhJ = ((b - bhh) A)_J, ncI = sum_J a_IJ.",
           "#pragma once", "", "namespace gx {", "namespace dop {"]
    A2 = A * A
    tiny = mpmath.mpf(10) ** -25  # what the published digits leave of a zero
    for i in range(2, 13):
        out.append(f"constexpr double nc{i} = {float(sum(A[i, j] for j in range(1, i))).hex()};")
        for j in range(1, i):
            if abs(A2[i, j]) > tiny:
                out.append(f"constexpr double n{i}_{j} = {float(A2[i, j]).hex()};")
    for name, row in (("nb", b * A), ("ner", er * A), ("nbh", bhh * A)):
        for j in range(1, 13):
            if abs(row[0, j]) > tiny:
                out.append(f"constexpr double {name}{j} = {float(row[0, j]).hex()};")
    out += ["}  // namespace dop", "}  // namespace gx", ""]
    print("\n".join(out))


if __name__ == "__main__":
    main()
