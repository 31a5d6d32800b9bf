"""What an orbit keeps of its extrema is ordinary memory, and its own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 33, 5000])
def test_statistics_are_not_kept_in_page_locked_memory(n):
    import torch

    import gala_gb300 as g
    from gala_gb300 import workloads as W

    pot = g.HernquistPotential(1e11, 1.0)
    orbits = [pot.integrate_orbit(W.mw_ics(n, seed=s), dt=1.0, n_steps=300, Integrator="leapfrog") for s in (1, 2)]
    first = [np.copy(orbits[0].pericenter()), np.copy(orbits[0].zmax(func=np.max))]
    orbits[1].pericenter()  # takes the block that the first call gave back
    kept = orbits[0]._ext_cache[False]
    assert not any(torch.from_numpy(kept[k]).is_pinned() for k in ("count", "sum", "min", "max"))
    again = [orbits[0].pericenter(), orbits[0].zmax(func=np.max)]
    assert all(np.array_equal(a, b, equal_nan=True) for a, b in zip(first, again))
