"""SCF value, gradient and density at the centre and where r underflows to it: gala's
sum of infinite terms (infinite where they have one sign, else NaN)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

Q = np.array([[0, 0, 0], [1e-200, 0, 0], [0, 1e-200, -1e-180], [1e-160, 0, 0], [3.0, 4.0, 5.0]], dtype=float).T.copy()


@pytest.mark.parametrize("nmax,lmax", [(0, 0), (1, 0), (3, 0), (23, 0), (0, 1), (4, 3), (12, 8)])
@pytest.mark.parametrize("signs", ["as drawn", "one sign", "the other"])
def test_density_at_the_centre(oracle, nmax, lmax, signs):
    import gala_gb300 as g
    from gala_gb300 import workloads as W

    S, T = W.scf_coefficients(nmax, lmax)[:2]
    if signs != "as drawn":  # C_n(-1) alternates in n
        S = np.abs(S) * (-1.0) ** np.arange(nmax + 1)[:, None, None] * (1 if signs == "one sign" else -1)
    pot = g.SCFPotential(m=1e12, r_s=20.0, Snlm=S, Tnlm=T)
    with np.errstate(all="ignore"):
        for name in ("energy", "density", "gradient"):
            ref, got = getattr(oracle, name)(pot, Q), getattr(pot, name)(Q)
            if name == "density" or lmax == 0:  # l > 0 at r = 0: NaN angles
                assert np.array_equal(np.isnan(got), np.isnan(ref)), name
            fin = np.isfinite(ref)
            assert np.allclose(got[fin], ref[fin], rtol=1e-10)
            inf = np.isinf(ref)
            assert np.array_equal(got[inf], ref[inf])
