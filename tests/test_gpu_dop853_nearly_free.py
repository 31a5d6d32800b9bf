"""Orbits whose accelerations are next to nothing, down to where their squares underflow:
straight lines, in each of the DOP853 orbit kernels."""
import numpy as np
import pytest

from tests.test_gpu_dop853_static import _stats

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rate,per_sm", [(0.0, 0), (0.0, 60), (1e-30, 0), (1e-30, 130)])
@pytest.mark.parametrize("kind", ["kepler", "nfw"])
def test_nearly_free_orbits(kind, rate, per_sm):
    import torch

    import gala_gb300 as g
    from gala_gb300 import workloads as W

    n = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + 37
    frame = g.ConstantRotatingFrame([0.0, 0.0, rate]) if rate else g.StaticFrame()
    w0, t = W.mw_ics(n, seed=4), np.arange(0, 20.5, 0.5)
    line = np.concatenate([w0[:3, None] + t[None, :, None] * w0[3:, None], np.repeat(w0[3:, None], len(t), axis=1)])
    for e in range(-120, -180, -3):
        pot = g.KeplerPotential(10.0 ** e) if kind == "kepler" else g.NFWPotential(5.4e11, 10.0 ** -e)
        w, s, c = _stats(pot, frame, w0, t)
        assert np.all(s == 1) and np.all(c[:, 3] == 0), e
        assert np.allclose(w, line, rtol=1e-13, atol=1e-13), e
