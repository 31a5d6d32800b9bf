"""A batch whose step size becomes NaN ends at once, with the return code and the
counters of gala's loop (eleven stages and a rejection per step up to nmax + 1), in
each of the DOP853 orbit kernels; the other batches of the call are not touched."""
import time

import numpy as np
import pytest

from tests.test_gpu_dop853_static import KW, _stats

pytestmark = pytest.mark.gpu


def _calls():
    """(frame rate, batch size, orbits as a multiple of the processors): few orbits
    one coordinate per lane, clusters of a static frame, one CTA per batch or two."""
    return [(0.0, 100, None), (0.03, 100, None), (0.0, 1, None), (0.0, 100, 60), (0.0, 256, 60), (0.0, 300, 10), (0.03, 100, 130),
            (0.03, 8, 130), (0.0, 8, 60)]


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("rate,nbatch,per_sm", _calls())
def test_nan_batch_ends_at_once(rate, nbatch, per_sm, bad):
    import torch

    import gala_gb300 as g
    from gala_gb300 import workloads as W

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = 2 * nbatch + 1 if per_sm is None else per_sm * sms + 7
    pot = W.mw_composite()
    frame = g.ConstantRotatingFrame([0.0, 0.0, rate]) if rate else g.StaticFrame()
    w0, t = W.mw_ics(n, seed=8), np.arange(0, 6.5, 0.5)
    ref, sr, cr = _stats(pot, frame, w0, t, nbatch=nbatch)
    assert np.all(sr == 1)
    b = min(1, len(sr) - 1)  # the batch of the orbit that is not finite
    w0[4, b * nbatch + nbatch // 3] = bad
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    w, s, c = _stats(pot, frame, w0, t, nbatch=nbatch)  # nmax: the default, 1,000,000 steps
    assert time.perf_counter() - t0 < 10.0  # rejected one by one they take about a minute
    others = np.arange(len(s)) != b
    assert np.array_equal(s[others], sr[others]) and np.array_equal(c[others], cr[others]) and s[b] == -2
    keep = np.repeat(others, nbatch)[:n]
    assert np.array_equal(w[..., keep], ref[..., keep])
    assert c[b].tolist() == [2 + 11 * 1000001, 1000001, 0, 0]


@pytest.mark.parametrize("rate", [0.0, 0.03])
@pytest.mark.parametrize("nmax", [1, 40])
def test_counters_are_those_of_the_loop(oracle, nmax, rate):
    """Against the oracle, which rejects the steps one by one."""
    import gala_gb300 as g
    from gala_gb300 import workloads as W

    pot, w0, t = W.mw_composite(), W.mw_ics(5, seed=8), np.arange(0, 6.5, 0.5)
    w0[0, 2] = np.nan
    frame = g.ConstantRotatingFrame([0.0, 0.0, rate]) if rate else g.StaticFrame()
    _, s, c = _stats(pot, frame, w0, t, nbatch=5, nmax=nmax)
    with np.errstate(all="ignore"):
        _, so, co = oracle.dop853(pot, w0, t, nbatch=5, nmax=nmax, frame=frame, **KW)
    assert np.array_equal(s, so) and np.array_equal(c, co)
