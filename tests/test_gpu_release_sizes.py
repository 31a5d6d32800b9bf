"""Leapfrog release systems larger than the declared largest release: up to three
members (eight where more than three are declared) they are integrated all the same,
with the bits of a call that declares them; larger ones get status -1."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("declared", [0, 1, 2, 3, 6])
def test_release_beyond_the_declared_size(declared):
    import torch

    import gala_gb300 as g
    from gala_gb300 import _abi
    from gala_gb300 import workloads as W
    from gala_gb300._device import ptr, stream_handle
    from gala_gb300.nbody import bodies_to_device, pack_bodies

    pot = W.mw_composite()
    counts = np.array([1, 2, 0, 7, 3, 2, 6, 1, 5, 4, 1, 2] * 5)
    S, R, P = 3, len(counts), int(counts.sum())
    rng = np.random.default_rng(5)
    bodies = np.stack([pack_bodies([g.PlummerPotential(1e5 * (s + 1), 0.05)]) for s in range(S)])
    prog = np.array([8., 0, 1, 0, 0.2, 0.05])
    nbody_w = np.broadcast_to(prog, (S, R, 1, 6)) * (1 + 0.01 * rng.normal(size=(S, R, 1, 6)))
    sw0 = prog * (1 + 0.01 * rng.normal(size=(S, P, 6)))
    off = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    rt = np.linspace(0., 90., R)

    def run(largest):
        d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (nbody_w, rt, off, sw0)]
        bd = bodies_to_device(bodies, torch.device("cuda"))
        out = torch.full((S, P, 6), -7., dtype=torch.float64, device="cuda")
        nb = torch.full((S, 1, 6), -7., dtype=torch.float64, device="cuda")
        status = torch.full((S, R), 9, dtype=torch.int32, device="cuda")
        _abi.call("gx_mockstream_leapfrog", pot.packed().for_device(), S, 1, ptr(bd), ptr(d[0]), R, ptr(d[1]), ptr(d[2]),
                  largest, ptr(d[3]), P, 100., 1., ptr(out), ptr(nb), ptr(status), stream_handle())
        return out.cpu().numpy(), nb.cpu().numpy(), status.cpu().numpy()

    out, nb, status = run(7)
    assert np.array_equal(status, np.broadcast_to(counts > 0, status.shape))
    most = 8 if declared > 2 else 3
    got, got_nb, got_status = run(declared)
    taken = counts + 1 <= most
    assert np.array_equal(got_status, np.broadcast_to(np.where(taken, counts > 0, -1), status.shape))
    rows = np.repeat(taken, counts)
    assert np.array_equal(got[:, rows], out[:, rows]) and np.all(got[:, ~rows] == -7.)
    assert np.array_equal(got_nb, nb)
