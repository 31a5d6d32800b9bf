"""The integer-pipe square root and quotient against the FP64 instructions on the
GPU, and the forms of the fixed-step kernels that rest on them: every component
type's orbits, and Ruth4's first sub-step where the gradient must and must not be
evaluated (gala multiplies it by zero, which a non-finite gradient survives)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _doubles(rng, n, kind):
    if kind == "any":  # every bit pattern
        return rng.integers(0, 2**64, n, dtype=np.uint64).view(np.float64)
    if kind == "edges":  # fractions at the ends, exponents around the limits of the integer path
        e = rng.choice(np.array([0, 1, 2, 510, 511, 512, 1022, 1023, 1024, 1534, 1535, 1536, 2045, 2046, 2047]), n).astype(np.uint64)
        f = rng.choice(np.array([0, 1, 2, 2**51, 2**52 - 2, 2**52 - 1], dtype=np.uint64), n)
        return ((rng.integers(0, 2, n).astype(np.uint64) << np.uint64(63)) | (e << np.uint64(52)) | f).view(np.float64)
    return rng.normal(size=n) * 10.0 ** rng.uniform(-30, 30, n)


@pytest.mark.parametrize("kind", ["any", "edges", "ordinary"])
def test_sqrt_and_quotient_have_ieee_bits(kind):
    import torch

    from gala_gb300 import _abi
    from gala_gb300._device import ptr, stream_handle

    rng = np.random.default_rng(7)
    n = 1 << 20
    x, y = _doubles(rng, n, kind), _doubles(rng, n, kind)
    xd, yd = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    out = torch.empty((6, n), dtype=torch.float64, device="cuda")
    _abi.call("gx_selfcheck_ipipe", ptr(xd), ptr(yd), n, ptr(out), stream_handle())
    sq, dv, sq_lib, dv_lib, s2, rs = out.cpu().numpy()
    assert np.array_equal(sq, sq_lib, equal_nan=True) and np.array_equal(dv, dv_lib, equal_nan=True)
    with np.errstate(all="ignore"):
        assert np.array_equal(np.signbit(dv[dv == 0]), np.signbit((x / y)[dv == 0]))
        ok = (x > 1e-290) & (x < 1e290)
        assert np.all(np.abs(s2[ok] - sq_lib[ok]) <= np.spacing(sq_lib[ok]))
        ref = 1.0 / np.sqrt(x[ok].astype(np.longdouble))
        assert np.all(np.abs(rs[ok] - ref) <= np.spacing(ref.astype(np.float64)))


@pytest.mark.parametrize("method", ["leapfrog", "ruth4"])
@pytest.mark.parametrize("where", ["plain", "singular", "shifted", "flat disk"])
def test_zero_coefficient_substep(oracle, method, where):
    """Orbits at ordinary places, on the singular point, in a shifted component
    and in a disk without thickness (regular descriptors and others)."""
    import gala_gb300 as g

    pot = {"plain": lambda: g.HernquistPotential(1e11, 1.0) + g.PlummerPotential(1e9, 0.3),
           "singular": lambda: g.HernquistPotential(1e11, 1.0),
           "shifted": lambda: g.HernquistPotential(1e11, 1.0, origin=[1.0, 2.0, 3.0]),
           "flat disk": lambda: g.MiyamotoNagaiPotential(1e11, 3.0, 0.0)}[where]()
    rng = np.random.default_rng(11)
    w0 = np.vstack([rng.uniform(-10, 10, (3, 45)), rng.normal(0, 0.1, (3, 45))])
    w0[:, 0] = 0.0                       # at rest on the origin
    w0[:, 1] = [1.0, 2.0, 3.0, 0, 0, 0]  # on the shifted centre
    w0[:3, 2] = [1e-40, 0, 0]            # below the range in which the gradient is taken as finite
    w0[2, 3] = w0[5, 3] = 0.0            # in the plane
    w0[:3, 4] = [1e40, 0, 0]
    t = np.arange(12) * 0.5
    with np.errstate(all="ignore"):
        ref = oracle.fixed(pot, w0, t, method)
    w = pot.integrate_orbit(w0, t=t, Integrator=method).w()
    if where == "flat disk":  # the power in its gradient does not round like the host's pow
        assert np.array_equal(np.isfinite(w), np.isfinite(ref))
        m = np.isfinite(ref)
        assert np.allclose(w[m], ref[m], rtol=1e-11, atol=1e-300)
    else:
        assert np.array_equal(w, ref, equal_nan=True)
    last = pot.integrate_orbit(w0, t=t, Integrator=method, save_all=False).w()
    assert np.array_equal(last[:, 0], w[:, -1], equal_nan=True)
