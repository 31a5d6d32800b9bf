"""The lanes of a warp without an orbit do not reach the results of those with one.

Copies of one orbit, a power of two of them, are one system whose sums are exact
multiples of the single orbit's, so the steps and the state are the same bits
whether a warp is filled by copies or by lanes without an orbit.  The scale radius
is one at which a point near the centre would take another form of the force."""
import numpy as np
import pytest

from tests.test_gpu_dop853_static import _stats

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rate", [0.0, 0.02])
@pytest.mark.parametrize("r_s", [15.6, 150.0])
def test_idle_lanes(r_s, rate):
    import gala_gb300 as g
    from gala_gb300 import workloads as W

    pot = g.NFWPotential(5e12, r_s) + g.MiyamotoNagaiPotential(6.8e10, 3.0, 0.28)
    frame = g.ConstantRotatingFrame([0.0, 0.0, rate]) if rate else g.StaticFrame()
    t = np.arange(0, 60.5, 0.5)
    w0 = W.mw_ics(3, seed=2)
    for i in range(3):
        one, s1, c1 = _stats(pot, frame, w0[:, [i]], t)
        for copies in (2, 4, 8, 16, 64):
            w, s, c = _stats(pot, frame, np.repeat(w0[:, [i]], copies, axis=1), t)
            assert np.array_equal(s, s1) and np.array_equal(c, c1)
            assert np.array_equal(w, np.repeat(one, copies, axis=2)), copies
