"""The sums of the extrema where a group of orbits is split over a cluster: 64 segments,
added by the CTA and then over the CTAs.  With about eight extrema in a segment that is
24 additions in a row, each off by 0.4 units of 2^-53 (rms) of a sum that grows evenly:
0.4 sqrt(24 / 3) 2^-53 = 1.26e-16 of the whole (72 in a row: 2.2e-16)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [33, 1000])
def test_rounding_of_the_sums(n):
    import torch

    import gala_gb300 as g

    nt = 5001
    u = torch.rand((6, n), generator=torch.Generator().manual_seed(n), dtype=torch.float64).cuda()
    T = torch.arange(nt, dtype=torch.float64, device="cuda")[:, None]
    r = (2 + 28 * u[0]) * (1 - (0.05 + 0.3 * u[1]) * torch.cos(0.2 * T + 6 * u[2]))
    w = torch.zeros((6, nt, n), dtype=torch.float64, device="cuda")
    w[0], w[1], w[2] = r * torch.cos(0.1 * T + 6 * u[3]), r * torch.sin(0.1 * T + 6 * u[3]), (0.1 + u[4]) * torch.cos(0.3 * T + 6 * u[5])
    o = g.Orbit.from_w(w, t=np.arange(nt) * 1.0)
    for kind in (o.pericenter, o.apocenter, o.zmax):
        each = kind(func=None)
        ref = np.array([np.sum(v.astype(np.longdouble)) / len(v) for v in each])
        err = (kind() - ref) / ref
        assert np.sqrt(np.mean(err.astype(np.float64) ** 2)) < 1.6e-16  # and the quotient's rounding
