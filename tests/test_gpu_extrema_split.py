"""Orbit extrema over every split of the groups of 32 orbits: a cluster per group,
whole rounds of one CTA per group, and a remainder.  A group's statistics do not
depend on how its time range is split except for the rounding of the sums: at most
one unit in the last place per extremum added (40 of them here)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("backwards", [False, True])
@pytest.mark.parametrize("n", [1, 32, 33, 9727, 9728, 9729, 19457])
def test_statistics_do_not_depend_on_the_split(n, backwards):
    import torch

    import gala_gb300 as g

    nt = 131
    t = np.arange(nt) * (-1.0 if backwards else 1.0)
    u = torch.rand((6, n), generator=torch.Generator().manual_seed(n), dtype=torch.float64).cuda()
    tt = torch.from_numpy(t).cuda()[:, None]
    r = 5 + 3 * torch.cos(tt * (0.3 + u[0]) + 6 * u[1])
    w = torch.zeros((6, nt, n), dtype=torch.float64, device="cuda")
    w[0], w[1], w[2] = r * torch.cos(tt * 0.2 + u[2]), r * torch.sin(tt * 0.2 + u[2]), torch.cos(tt * u[3] + 6 * u[4])
    whole = g.Orbit.from_w(w, t=t)._extrema_run(False, 0)
    for a in sorted({0, max(n - 40, 0), n // 2}):
        b = min(a + 40, n)
        part = g.Orbit.from_w(w[:, :, a:b].contiguous(), t=t)._extrema_run(False, 0)
        for k in ("count", "min", "max"):
            assert np.array_equal(whole[k][:, a:b], part[k], equal_nan=True)
        assert np.allclose(whole["sum"][:, a:b], part["sum"], rtol=40 * 2.3e-16, atol=0)
