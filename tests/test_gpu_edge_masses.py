"""Masses at the edges of the number range in each component of a disk-bulge-halo
composite: the straight-run gradients give the bits of the component loop, which the
same composite with a null component takes, in calls on both sides of the lines
between the kernels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MASSES = {"zero": 0.0, "minus zero": -0.0, "nan": np.nan, "inf": np.inf, "subnormal": 1e-310, "tiny": 1e-300, "small": 1e-145,
          "below the quotient's range": 1e-144, "huge": 1e300, "large": 1e160, "negative": -3e9}


def _pair(order, pos, mass):
    import gala_gb300 as g

    m = [1.7e9, 5e9, 6.8e10, 5.4e11]
    m[pos] = mass
    c = [g.HernquistPotential(m[0], 0.07), g.HernquistPotential(m[1], 1.0), g.MiyamotoNagaiPotential(m[2], 3.0, 0.28),
         g.NFWPotential(m[3], 15.6)]
    c = [c[i] for i in order]
    pot = c[0] + c[1] + c[2] + c[3]
    return pot, c[0] + c[1] + c[2] + c[3] + g.NullPotential()


@pytest.mark.parametrize("mass", MASSES)
@pytest.mark.parametrize("pos", [0, 1, 2, 3])
@pytest.mark.parametrize("order", [(0, 1, 2, 3), (1, 0, 2, 3), (2, 0, 1, 3)])
def test_masses_at_the_edges_of_the_range(oracle, order, pos, mass):
    import torch

    from gala_gb300 import workloads as W
    from gala_gb300.batch import BatchIntegrator
    from gala_gb300.nbody import BODY_DTYPE, integrate_systems_leapfrog

    pot, loop = _pair(order, pos, MASSES[mass])
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = 160 * sms + 33
    w0 = W.mw_ics(n, seed=5)
    w0[:3, 3], w0[:3, 12] = [0.3, 0.0, 0.0], [0.0, 0.0, 2.0]
    same = lambda a, b: np.array_equal(a, b, equal_nan=True)  # noqa: E731

    q = w0[:3, :64].copy()
    grad = pot.gradient(q)
    assert same(grad, loop.gradient(q))
    with np.errstate(all="ignore"):
        ref = oracle.gradient(pot, q)
    fin = np.isfinite(ref)
    assert same(np.isfinite(grad), fin) and np.allclose(grad[fin], ref[fin], rtol=1e-12, atol=0)

    t = np.arange(4) * 0.5
    for k in (21, 32 * sms, 32 * sms + 9):
        for method in ("leapfrog", "ruth4"):
            a, b = (p.integrate_orbit(w0[:, :k], t=t, Integrator=method, save_all=False).w() for p in (pot, loop))
            assert same(a, b), (k, method)
    ns, m = np.full(n, 3), (np.arange(n) % 2).astype(np.int32)
    for k in (50, n):
        a, b = (BatchIntegrator(p, w0[:, :k], ns[:k], np.full(k, 0.5), m[:k], precision="fp64").run().cpu().numpy() for p in (pot, loop))
        assert same(a, b), k
    systems = np.ascontiguousarray(w0[:, :90].T.reshape(30, 3, 6))
    a, b = (integrate_systems_leapfrog(p, np.zeros((30, 0), dtype=BODY_DTYPE), systems, t).cpu().numpy() for p in (pot, loop))
    assert same(a, b)
