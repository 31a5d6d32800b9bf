"""The static-frame DOP853 kernel (a cluster of one-warp CTAs per batch) in populations
that are above the line of the kernel for few orbits: every size of a cluster, partial
last batches (CTAs of a cluster without an orbit), against the oracle and against the
general kernel, which the same call takes in a frame that rotates at rate zero.
Tolerances as in test_gpu_dop853_static.py; every size is checked to take the kernel
that it is meant for."""
import ctypes as C

import numpy as np
import pytest

from tests.test_gpu_dop853_static import KW, _close, _stats

pytestmark = pytest.mark.gpu

GENERAL, CLUSTER, AXIS = 0, 1, 2


def _form(pot, frame, n, nbatch):
    import gala_gb300 as g
    from gala_gb300 import _abi

    form = C.c_int32(-1)
    _abi.call("gx_dop853_form", pot.packed().for_device(), g.Hamiltonian(pot, frame)._frame_ref(), n, nbatch, C.addressof(form))
    return form.value


def _population(nbatch, warps_per_sm, last):
    """Orbits in batches of nbatch, the last one of `last`, of more than warps_per_sm
    warps (eight orbits each) per processor."""
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return (warps_per_sm * sms // ((nbatch + 7) // 8) + 1) * nbatch + last


def test_lines_between_the_kernels():
    import gala_gb300 as g
    from gala_gb300 import workloads as W

    mw, static, rot = W.mw_composite(), g.StaticFrame(), g.ConstantRotatingFrame([0.0, 0.0, 0.02])
    shifted = g.HernquistPotential(1e11, 1.0, origin=[0.5, 0.2, -0.1]) + g.NFWPotential(5.4e11, 15.6)
    for nb in (17, 100, 256):
        assert _form(mw, static, nb, nb) == _form(mw, rot, nb, nb) == AXIS
        n = _population(nb, 6, 1)
        assert _form(mw, static, n, nb) == CLUSTER and _form(mw, rot, n, nb) == AXIS and _form(shifted, rot, n, nb) == GENERAL
        assert _form(mw, rot, _population(nb, 14, 1), nb) == GENERAL
    assert _form(mw, static, 7, 100) == AXIS and _form(mw, static, 1000, 16) == GENERAL and _form(mw, static, 1000, 257) == GENERAL
    assert _form(W.scf_potential(4, 3), static, 100, 100) == CLUSTER and _form(W.scf_potential(4, 3), rot, 100, 100) == GENERAL


@pytest.mark.parametrize("nbatch,last", [(17, 3), (32, 1), (33, 33), (64, 33), (96, 5), (100, 11), (100, 97), (128, 64), (160, 129),
                                         (192, 1), (224, 220), (256, 31), (256, 255)])
def test_every_size_of_a_cluster_against_oracle(oracle, nbatch, last):
    import gala_gb300 as g
    from gala_gb300 import workloads as W

    mw, n = W.mw_composite(), _population(nbatch, 6, last)
    assert _form(mw, g.StaticFrame(), n, nbatch) == CLUSTER
    w0, t = W.mw_ics(n, seed=nbatch), np.arange(0, 50.5, 0.5)
    w, s, c = _stats(mw, g.StaticFrame(), w0, t, nbatch=nbatch)
    assert np.all(s == 1)
    for b in (0, len(s) // 2, len(s) - 1):
        sl = slice(b * nbatch, min((b + 1) * nbatch, n))
        ref, so, co = oracle.dop853(mw, w0[:, sl], t, nbatch=nbatch, **KW)
        assert so[0] == 1 and co[0, 1:].tolist() == c[b, 1:].tolist()  # steps tried, accepted, rejected
        assert _close(w[:, :, sl], ref)


@pytest.mark.parametrize("opts", [dict(), dict(out_stride=7), dict(save_all=0), dict(dt_max=0.7), dict(nstiff=1), dict(nmax=20),
                                  dict(back=True), dict(same_times=True)])
@pytest.mark.parametrize("name", ["dbh", "one sphere", "plain", "shifted", "triaxial", "scf", "wide", "centre"])
def test_against_general_kernel_above_the_line(name, opts):
    import gala_gb300 as g
    from gala_gb300 import workloads as W

    nfw = dict(m=5.4e11, r_s=15.6)

    def wide():  # more components than the descriptor holds by value
        pot = g.CCompositePotential()
        for k in range(20):
            pot[f"c{k}"] = g.PlummerPotential(5e9, 1.0 + 0.1 * k, origin=[0.05 * k, 0.0, -0.02 * k])
        return pot

    pot = {"dbh": W.mw_composite, "one sphere": lambda: g.NFWPotential(**nfw) + g.MiyamotoNagaiPotential(6.8e10, 3.0, 0.28) + g.HernquistPotential(5e9, 1.0),
           "plain": lambda: g.PlummerPotential(1e11, 2.0) + g.KeplerPotential(1e9),
           "shifted": lambda: g.HernquistPotential(1e11, 1.0, origin=[0.5, 0.2, -0.1]) + g.NFWPotential(**nfw),
           "triaxial": lambda: g.NFWPotential(b=0.9, c=0.8, **nfw) + g.MiyamotoNagaiPotential(6.8e10, 3.0, 0.28),
           "scf": lambda: W.scf_potential(4, 3), "wide": wide, "centre": W.mw_composite}[name]()
    n = 153 if name in ("scf", "wide") else _population(100, 14, 53)
    assert _form(pot, g.StaticFrame(), n, 100) == CLUSTER and _form(pot, g.ConstantRotatingFrame([0.0] * 3), n, 100) == GENERAL
    w0 = W.mw_ics(n, seed=9)
    if name == "centre":  # radial orbits through the region that the straight run hands to the general form
        w0[3:] *= 0.05
    opts = dict(opts)
    t = np.arange(0, 40.5, 0.5)
    if opts.pop("back", False):
        t = -t
    if opts.pop("same_times", False):  # h0 = 0: the starting step is estimated
        t = np.concatenate([t[:1], t])
    a, sa, ca = _stats(pot, g.StaticFrame(), w0, t, **opts)
    b, sb, cb = _stats(pot, g.ConstantRotatingFrame([0.0, 0.0, 0.0]), w0, t, **opts)
    for k in (0, len(sa) - 1):  # the first batch and the partial last
        sl = slice(100 * k, min(100 * (k + 1), n))
        assert sa[k] == sb[k] and np.array_equal(ca[k], cb[k])
        # close passages of the centre amplify a last-bit difference further
        assert _close(a[..., sl], b[..., sl], 1e-9 if name == "centre" else 1e-12)
