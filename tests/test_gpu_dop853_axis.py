"""DOP853 with one coordinate per lane (few orbits) against the kernels that larger
calls take: the batches of a call are independent, so the first two batches of a
large call and a call of those orbits alone are the same systems.

Sums run in another order and the force's squares are rounded once more or less:
a few units in the last place per step, as between the kernels and the oracle
(1e-12 of the state over these spans; 1e-9 where close passages of the centre
amplify it).  Step counts and return codes are equal."""
import numpy as np
import pytest

from tests.test_gpu_dop853_static import _close, _stats

pytestmark = pytest.mark.gpu


def _pot(name):
    import gala_gb300 as g
    from gala_gb300 import workloads as W

    nfw = dict(m=5.4e11, r_s=15.6)
    return {"dbh": W.mw_composite, "bar": lambda: g.PlummerPotential(1e10, 0.5) + g.MiyamotoNagaiPotential(6.8e10, 3.0, 0.28)
            + g.NFWPotential(b=0.9, c=0.8, **nfw), "shifted": lambda: g.HernquistPotential(1e11, 1.0, origin=[0.5, 0.2, -0.1])
            + g.NFWPotential(c=0.7, **nfw) + g.KeplerPotential(1e9), "centre": W.mw_composite}[name]()


@pytest.mark.parametrize("opts", [dict(), dict(out_stride=7), dict(save_all=0), dict(nstiff=1), dict(nmax=20), dict(back=True),
                                  dict(same_times=True), dict(nbatch=250), dict(nbatch=17)])
@pytest.mark.parametrize("rotating", [False, True])
@pytest.mark.parametrize("name", ["dbh", "bar", "shifted", "centre"])
def test_few_orbits_equal_the_first_batches_of_many(name, rotating, opts):
    import torch

    import gala_gb300 as g
    from gala_gb300 import workloads as W

    pot = _pot(name)
    frame = g.ConstantRotatingFrame([0.01, -0.02, 0.04]) if rotating else g.StaticFrame()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    opts = dict(opts)
    nb = opts.get("nbatch", 100)
    w0 = W.mw_ics(120 * sms, seed=9)
    if name == "centre":
        w0[3:] *= 0.05
    t = np.arange(0, 40.5, 0.5)
    if opts.pop("back", False):
        t = -t
    if opts.pop("same_times", False):
        t = np.concatenate([t[:1], t])
    b, sb, cb = _stats(pot, frame, w0, t, **opts)
    a, sa, ca = _stats(pot, frame, w0[:, :2 * nb], t, **opts)
    assert np.array_equal(sa, sb[:2]) and np.array_equal(ca, cb[:2])
    assert _close(a, b[..., :2 * nb], 1e-9 if name == "centre" else 1e-12)


@pytest.mark.parametrize("n", [1, 7, 8, 9, 63, 64, 65, 128, 129, 256])
def test_every_size_of_a_batch(oracle, n):
    """One batch of 1 to 32 warps, in clusters of 1 to 8 CTAs."""
    import gala_gb300 as g
    from gala_gb300 import workloads as W

    mw, w0 = W.mw_composite(), W.mw_ics(n, seed=n)
    t = g.parse_time_specification(dt=0.5, n_steps=120)
    H = g.Hamiltonian(mw, g.ConstantRotatingFrame([0.0, 0.0, 0.03]))
    w = H.integrate_orbit(w0, t=t, Integrator="dop853", Integrator_kwargs=dict(atol=1e-12, rtol=1e-10, nbatch=256)).w()
    ref, st, _ = oracle.dop853(mw, w0, t, nbatch=256, atol=1e-12, rtol=1e-10, frame=H.frame)
    assert np.all(st == 1) and _close(w.reshape(ref.shape), ref)
