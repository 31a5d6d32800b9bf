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


@pytest.mark.parametrize("extra,shapes", [(0, 2), (1, None)])
def test_autotune_times_the_shapes_that_differ(tmp_path, monkeypatch, extra, shapes):
    """Four lanes per orbit ignore block and CTA count: only the chunk is searched, and the
    record keeps the block and CTA count that larger batches were tuned to."""
    import json

    import torch

    import gala_gb300.batch as B
    from gala_gb300 import workloads as W

    cache = tmp_path / "autotune.json"
    monkeypatch.setattr(B, "CACHE", cache)
    n = 32 * torch.cuda.get_device_properties(0).multi_processor_count + extra
    args = (_pot("plummer"), W.mw_ics(n, seed=3), np.full(n, 4), np.full(n, 0.5), np.zeros(n, dtype=np.int32))
    key = B.BatchIntegrator(*args, precision="fp64")._cache_key()
    tuned = {"block": 64, "ctas_per_sm": 8, "chunk": 64}
    cache.write_text(json.dumps({key: tuned}))
    b = B.BatchIntegrator(*args, precision="fp64")
    best = b.autotune(work_fraction=1.0, reps=1)
    record = json.loads(cache.read_text())[key]
    assert record == best and len(b.tune_results) == (shapes or len(B.SEARCH["fp64"]))
    if shapes:
        assert {k: best[k] for k in ("block", "ctas_per_sm")} == {k: tuned[k] for k in ("block", "ctas_per_sm")}
