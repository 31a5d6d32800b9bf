"""Which form an FP64 batch takes by its size: four lanes per orbit only where even
lengths do not lose by it (one block of 32 orbits per processor for the component
loop, two for a Hernquist sphere), or spread ones gain enough (straight-run
composites); both forms give the same bits at the lines."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pot(name):
    import gala_gb300 as g
    from gala_gb300 import workloads as W

    return {"sphere": lambda: g.HernquistPotential(1e11, 1.0), "mw": W.mw_composite, "plummer": lambda: g.PlummerPotential(1e11, 1.0),
            "shifted": lambda: g.HernquistPotential(1e11, 1.0, origin=[0.3, 0.2, 0.1]) + g.NFWPotential(5.4e11, 15.6, c=0.7)}[name]()


@pytest.mark.parametrize("name,per_sm", [("sphere", 64), ("mw", 160), ("plummer", 32), ("shifted", 32)])
def test_lines_between_the_forms(name, per_sm):
    import torch

    from gala_gb300 import _abi
    from gala_gb300 import workloads as W
    from gala_gb300.batch import BatchIntegrator

    pot = _pot(name)
    line = per_sm * torch.cuda.get_device_properties(0).multi_processor_count
    lanes = C.c_int32()
    for n, want in ((1, 4), (line, 4), (line + 1, 1), (10 * line, 1)):
        _abi.call("gx_batch_fp64_lanes", pot.packed().for_device(), n, C.addressof(lanes))
        assert lanes.value == want, n
    w0, ns, m = W.mw_ics(line + 1, seed=3), np.full(line + 1, 4), (np.arange(line + 1) % 2).astype(np.int32)
    a, b = (BatchIntegrator(pot, w0[:, :n], ns[:n], np.full(n, 0.5), m[:n], precision="fp64").run().cpu().numpy() for n in (line, line + 1))
    assert np.array_equal(a, b[:, :line])
