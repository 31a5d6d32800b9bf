"""Fixed-step kernels with one coordinate per lane (few orbits) against the oracle
and, bit for bit, against the one-lane kernels that larger calls take; the uneven
batch in both forms; Leapfrog n-body systems with one body per lane."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pots():
    import gala_gb300 as g
    from gala_gb300 import workloads as W

    nfw = dict(m=5.4e11, r_s=15.6)
    return {"sphere": g.HernquistPotential(1e11, 1.0), "plummer": g.PlummerPotential(1e11, 1.0), "mw": W.mw_composite(),
            "disk first": g.MilkyWayPotential(),
            "one sphere": g.MiyamotoNagaiPotential(6.8e10, 3.0, 0.28) + g.HernquistPotential(5e9, 1.0) + g.NFWPotential(**nfw),
            "halo first": g.NFWPotential(**nfw) + g.MiyamotoNagaiPotential(6.8e10, 3.0, 0.28) + g.HernquistPotential(5e9, 1.0),
            "mixed": g.KeplerPotential(1e9) + g.NFWPotential(b=0.9, c=0.8, **nfw) + g.NFWPotential(c=0.7, **nfw)
            + g.HernquistPotential(1e10, 1.0, origin=[0.3, 0.2, 0.1])}


@pytest.mark.parametrize("method", ["leapfrog", "ruth4"])
@pytest.mark.parametrize("name", ["sphere", "plummer", "mw", "disk first", "one sphere", "halo first", "mixed"])
def test_one_coordinate_per_lane_has_the_bits_of_one_lane_per_orbit(oracle, name, method):
    from gala_gb300 import workloads as W

    import torch

    pot = _pots()[name]
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    w0 = W.mw_ics(32 * sms + 1, seed=21)
    w0[:, 3] *= 0.02                    # near the centre: the straight run declines it
    w0[:, 5] = [0, 0, 0, 0.1, 0, 0.05]  # on it
    w0[0, 8] = np.nan
    t = np.arange(25) * 0.7
    full = pot.integrate_orbit(w0, t=t, Integrator=method).w()          # one lane per orbit
    for n in (1, 7, 8, 9, 33, 32 * sms):
        few = pot.integrate_orbit(w0[:, :n], t=t, Integrator=method).w().reshape(6, len(t), n)
        assert np.array_equal(few, full[:, :, :n], equal_nan=True)
        last = pot.integrate_orbit(w0[:, :n], t=t, Integrator=method, save_all=False).w().reshape(6, n)
        assert np.array_equal(last, full[:, -1, :n], equal_nan=True)
    ok = [0, 1, 2, 4, 6, 7]  # ordinary orbits against gala's arithmetic
    with np.errstate(all="ignore"):
        ref = oracle.fixed(pot, w0[:, ok], t, method)
    assert np.allclose(full[:, :, ok], ref, rtol=1e-11, atol=1e-13)


@pytest.mark.parametrize("n", [5, 1000, 32])
@pytest.mark.parametrize("name", ["sphere", "mw", "disk first", "mixed"])
def test_uneven_batch_small_and_large_forms(oracle, name, n):
    """The same orbits alone (four lanes per orbit) and inside a batch of more than
    160 per SM (one lane per orbit); the order of the batch does not matter."""
    import torch

    from gala_gb300 import workloads as W
    from gala_gb300.batch import BatchIntegrator

    pot = _pots()[name]
    rng = np.random.default_rng(n)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    big = 160 * sms + 77
    w0, ns = W.mw_ics(big, seed=4), rng.integers(0, 40, big)
    dt, m = rng.choice(np.array([0.1, 0.5, 1.0]), big), rng.integers(0, 2, big).astype(np.int32)
    w0[:, 2] = [0, 0, 0, 0.1, 0, 0.05]
    many = BatchIntegrator(pot, w0, ns, dt, m, precision="fp64").run().cpu().numpy()[:, :n]
    for cfg in (None, dict(block=32, ctas_per_sm=1, chunk=64), dict(block=128, ctas_per_sm=2, chunk=32)):
        b = BatchIntegrator(pot, w0[:, :n], ns[:n], dt[:n], m[:n], precision="fp64", config=cfg)
        few = b.run().cpu().numpy()
        assert np.array_equal(few, many, equal_nan=True)
        assert bool(b.completed().all())
        # an order of both integrators in every warp
        b.order = torch.cat([torch.randperm(n, device="cuda").to(torch.int32),
                             torch.full((b.order.numel() - n,), -1, dtype=torch.int32, device="cuda")])
        assert np.array_equal(b.run().cpu().numpy(), many, equal_nan=True)
    with np.errstate(all="ignore"):
        ref = oracle.batch_fixed(pot, w0[:, :n], ns[:n], dt[:n], m[:n])
    ok = np.isfinite(ref).all(axis=0)
    ok[2:3] = False
    assert np.allclose(many[:, ok], ref[:, ok], rtol=1e-11, atol=1e-13)


@pytest.mark.parametrize("nbody,nparticles", [(0, 1), (1, 1), (1, 3), (2, 2), (3, 5), (8, 8)])
def test_leapfrog_bodies_one_per_lane(oracle, nbody, nparticles):
    """Bodies move in gala's order within a step: j < k already moved, j > k not."""
    import gala_gb300 as g
    from gala_gb300 import workloads as W
    from gala_gb300.nbody import BODY_DTYPE, integrate_systems_leapfrog, pack_bodies

    mw = W.mw_composite()
    S = 37
    rng = np.random.default_rng(nparticles)
    w0 = np.ascontiguousarray(W.mw_ics(S * nparticles, seed=6).T.reshape(S, nparticles, 6))
    pots = [[g.PlummerPotential(m=float(rng.uniform(1e8, 1e10)), b=0.5) for _ in range(nbody)] for _ in range(S)]
    bodies = pack_bodies(pots) if nbody else np.zeros((S, 0), dtype=BODY_DTYPE)
    t = np.arange(40) * 1.0
    w = integrate_systems_leapfrog(mw, bodies, w0, t).cpu().numpy()
    last = integrate_systems_leapfrog(mw, bodies, w0, t, save_all=False).cpu().numpy()
    assert np.array_equal(last, w[:, -1])
    for s in (0, 17, S - 1):
        ref = oracle.leapfrog_nbody(mw, bodies[s], nbody, w0[s], t)
        assert np.allclose(w[s], np.asarray(ref).reshape(w[s].shape), rtol=1e-11, atol=1e-13)
