"""GPU: the captured training step takes every input of a call from that call.

The step is captured once per batch size; rows, targets, loss weights, the index array, the learning rate and Adam's
step count are read from device memory. A network that has trained before on other inputs and is then reset to some
parameters (which clears its moments and step count) must give the same bits as a network that never trained: the
gradients' partial sums are added in a fixed order. The reported loss alone is added by atomics over at most 192
blocks of a step: 2^-24 for each addition, relative to a sum of positive terms.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    import torch
    from tardiis_and_claritas_gb300.build_ext import build
    build()
    return torch


def _data(torch, rows, seed):
    rng = np.random.default_rng(seed)
    return [torch.from_numpy(a.astype(np.float32)).cuda() for a in
            (rng.normal(size=(rows, 6)), rng.normal(size=(rows, 3)), rng.uniform(0.5, 2.0, size=(rows, 3)))]


# batch, index positions, loss weights, learning rate; the warm-up call before differs from each in everything
CALLS = [(512, 700, False, 1e-3), (512, 2999, True, 5e-4), (256, 900, False, 1e-3), (512, 512, True, 2e-3),
         (512, 1024, False, 2e-3)]


@pytest.mark.parametrize("batch,rows,weighted,lr", CALLS)
@pytest.mark.parametrize("warm_batch", [256, 512])  # with and without a step captured anew
def test_a_trained_network_steps_as_a_new_one(torch_cuda, batch, rows, weighted, lr, warm_batch):
    torch = torch_cuda
    from tardiis_and_claritas_gb300 import lib as L
    x, t, w = _data(torch, 3000, 5)
    x2, t2, w2 = _data(torch, 1500, 6)
    idx = torch.from_numpy(np.random.default_rng(7).permutation(3000)[:rows].astype(np.int32)).cuda()
    idx2 = torch.from_numpy(np.random.default_rng(8).permutation(1500).astype(np.int32)).cuda()
    used, new = (L.Network(0, max_batch=512, seed=2) for _ in range(2))
    start = new.get_params()
    used.set_loss_weights(0 if weighted else w2.data_ptr())
    used.train(x2.data_ptr(), t2.data_ptr(), idx2.data_ptr(), 1500, warm_batch, 7e-3)
    used.set_params(start)
    losses = []
    for net in (used, new):
        net.set_loss_weights(w.data_ptr() if weighted else 0)
        losses.append(net.train(x.data_ptr(), t.data_ptr(), idx.data_ptr(), rows, batch, lr))
    a, b = used.get_params(), new.get_params()
    np.testing.assert_array_equal(a, b)
    steps = rows // batch
    assert np.abs(b - start).max() > 0.5 * lr  # Adam's first step moves a weight by its learning rate
    assert np.abs(b - start).max() < 2.0 * lr * steps
    assert abs(losses[0] - losses[1]) <= 192 * steps * 2.0**-24 * losses[1]
    for net in (used, new):
        net.close()
