"""The training products at batches around the edges of their tiles (128 rows, slabs of
16, shares of the batch for the weight gradients), with 16-byte aligned buffers and with
buffers that start 4 bytes further on, against the FP64 network."""
import ctypes as C

import numpy as np
import pytest

from oracle import mlp_oracle as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("batch", [1, 16, 127, 129, 1000])
def test_training_step_matches_fp64(batch, offset):
    import torch

    from gala_gb300 import _abi

    lib = _abi.load()
    rng = np.random.default_rng(100 * batch + offset)
    p = (rng.normal(0, 0.08, lib.gx_mlp_param_count())).astype(np.float32)
    X = rng.uniform(-1, 1, (batch, 3)).astype(np.float32)
    ys = rng.normal(0, 0.3, batch).astype(np.float32)
    Gs = rng.normal(0, 0.3, (batch, 3)).astype(np.float32)

    def held(n):
        return torch.full((n + offset,), float("nan"), dtype=torch.float32, device="cuda")[offset:]

    params = held(len(p))
    params.copy_(torch.from_numpy(p))
    grads = held(len(p))
    ws = held(int(lib.gx_mlp_train_workspace_floats(batch)))
    loss = torch.zeros(2, dtype=torch.float32, device="cuda")
    Xd, yd, Gd = (torch.from_numpy(a).cuda() for a in (X, ys, Gs))
    _abi.call("gx_mlp_train_step", params.data_ptr(), grads.data_ptr(), Xd.data_ptr(), yd.data_ptr(), Gd.data_ptr(), None,
              batch, C.c_float(0.8), C.c_float(1.2), ws.data_ptr(), loss.data_ptr(), None)
    L, want = M.loss_and_grad(p.astype(np.float64), X.astype(np.float64), ys.astype(np.float64), Gs.astype(np.float64), 0.8, 1.2)
    got = grads.cpu().numpy()
    # sums of 256 products through eight layers and of `batch` terms, all in FP32: a few
    # 1e-6 of the largest entry; a lost row of the batch is 1/batch, a lost slab 1/16
    assert np.max(np.abs(got - want)) <= 5e-5 * np.abs(want).max()
    total = 0.8 * loss[0].item() + 1.2 * loss[1].item()
    assert abs(total - L) <= 2e-5 * abs(L)
