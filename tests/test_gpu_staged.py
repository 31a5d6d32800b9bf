"""Potential evaluations of small host arrays (read and written in place in a
page-locked block) against the device path, at both sides of the size line and
for every layout the call takes."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [0, 1, 31, 257, 10922, 10923])
@pytest.mark.parametrize("kind", ["energy", "gradient", "density"])
def test_staged_equals_device(kind, n):
    import torch

    from gala_gb300 import workloads as W

    pot, q = W.mw_composite(), W.mw_ics(max(n, 1), seed=3)[:3, :n]
    f = getattr(pot, kind)
    ref = f(torch.from_numpy(np.ascontiguousarray(q)).cuda())
    assert np.array_equal(f(q), ref) and f(q).shape == ref.shape
    if n > 1:
        assert np.array_equal(f(np.asfortranarray(q)), ref)        # other strides
        assert np.array_equal(f(q[:, ::-1]), ref[..., ::-1])
        assert np.array_equal(f(q[:, :1].reshape(3, 1, 1)), ref[..., :1].reshape(ref[..., :1].shape + (1,)))
        assert np.array_equal(f(q[:, 0]), ref[..., 0])
        first = f(q)
        keep = first.copy()
        f(q * 1.5)
        assert np.array_equal(first, keep)  # a result is the caller's own


def test_staged_on_streams_and_threads():
    import torch

    from gala_gb300 import workloads as W

    pot, q = W.mw_composite(), W.mw_ics(64, seed=3)[:3]
    ref, bad = pot.gradient(q), []

    def work(k):
        with torch.cuda.stream(torch.cuda.Stream()):
            for i in range(50):
                if not np.array_equal(pot.gradient(np.roll(q, k + i, axis=1)), np.roll(ref, k + i, axis=1)):
                    bad.append((k, i))

    ts = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not bad
