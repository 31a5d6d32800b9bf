"""The SCF sums (gala_gb300/csrc/gx_scf.cuh) against the oracle at the ends of
their range: no radial or no angular terms, the largest orders, sparse
coefficients, points from deep inside to far out, and the pole.

Tolerance: the recurrences run over at most 24 and 16 terms and the sums over
24 x 136 terms of either sign, each rounding once: about 1e-13 of the largest
term; 1e-11 of the point's own scale leaves room for cancellation between terms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pot(nmax, lmax, sparse):
    import gala_gb300 as g

    rng = np.random.default_rng(17)
    n, l, m = np.ogrid[:nmax + 1, :lmax + 1, :lmax + 1]
    amp = np.where(m <= l, np.exp(-0.5 * n) * (l + 1.0) ** -2, 0.0)
    S, T = rng.normal(size=amp.shape) * amp, rng.normal(size=amp.shape) * amp * (m > 0)
    if sparse:
        keep = rng.random(amp.shape) < 0.2
        S, T = S * keep, T * keep
    S[0, 0, 0] = 1.0
    return g.SCFPotential(m=1e12, r_s=20.0, Snlm=S, Tnlm=T)


def _points(n=300):
    rng = np.random.default_rng(23)
    u = rng.normal(size=(3, n))
    u /= np.linalg.norm(u, axis=0)
    u[:, np.hypot(u[0], u[1]) < 0.05] = np.array([[0.6], [0.0], [0.8]])  # the oracle's sin theta loses digits nearer the pole
    return u * np.exp(rng.uniform(np.log(0.02), np.log(2000.0), n))


@pytest.mark.parametrize("sparse", [False, True])
@pytest.mark.parametrize("nmax,lmax", [(0, 0), (1, 0), (0, 1), (1, 1), (2, 3), (12, 8), (23, 15)])
def test_scf_against_oracle(oracle, nmax, lmax, sparse):
    pot, q = _pot(nmax, lmax, sparse), _points()
    r = np.linalg.norm(q, axis=0)
    # the sizes of the monopole's value and density at each point
    phi0, rho0 = pot.G * 1e12 / (r + 20.0), 1e12 * 20.0 / (2 * np.pi * r * (r + 20.0) ** 3)
    assert np.all(np.abs(pot.energy(q) - oracle.energy(pot, q)) <= 1e-11 * phi0)
    assert np.all(np.abs(pot.density(q) - oracle.density(pot, q)) <= 1e-9 * rho0)  # terms weighted by K_nl <= 1,500
    got, ref = pot.gradient(q), oracle.gradient(pot, q)
    assert np.all(np.abs(got - ref) <= 1e-11 * np.linalg.norm(ref, axis=0))


@pytest.mark.parametrize("nmax,lmax", [(2, 0), (2, 2)])
def test_scf_on_the_pole(oracle, nmax, lmax):
    """gala divides by sin theta there; which components survive is kept."""
    pot, q = _pot(nmax, lmax, False), np.array([[0.0, 0.0], [0.0, 0.0], [5.0, -7.0]])
    with np.errstate(all="ignore"):
        ref = oracle.gradient(pot, q)
    got = pot.gradient(q)
    assert np.array_equal(np.isfinite(got), np.isfinite(ref))
    assert np.allclose(pot.energy(q), oracle.energy(pot, q), rtol=1e-12, atol=0)
