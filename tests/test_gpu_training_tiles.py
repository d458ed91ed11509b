"""GPU: the training kernels at the edges of their tiles.

The tensor-core product takes 128 rows and 64 columns per CTA and K in a ring of four 64-wide stages; the small
gradient reductions take 256 batch rows per block, the thin layers 16. The products are checked against a PyTorch
FP32 product of the same BF16 values (only the summation order differs: 1e-5 relative, 1e-4 sqrt(K) absolute for
unit normals, as for the other sizes), the gradients against the numpy oracle with its BF16 roundings (2e-2 of
the norm of every parameter block, the bound of the other batch sizes).
"""
from __future__ import annotations

import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), "..", "oracle"))
import mlp_reference as M  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    import torch
    from tardiis_and_claritas_gb300.build_ext import build
    build()
    return torch


@pytest.mark.parametrize("rows,K", [(1, 64), (129, 320), (128, 576), (257, 1024)])
def test_product_ring_of_stages(torch_cuda, rows, K):
    torch = torch_cuda
    from tardiis_and_claritas_gb300 import lib as L
    g = torch.Generator(device="cpu").manual_seed(rows * 7 + K)
    a = torch.randn(rows, K + 8, generator=g).to(torch.bfloat16).cuda()[:, :K]  # a leading dimension of its own
    b = torch.randn(256, K, generator=g).to(torch.bfloat16).cuda()
    c = torch.full((rows, 260), float("nan"), dtype=torch.float32, device="cuda")
    L.bf16_gemm_n256(a.data_ptr(), K + 8, b.data_ptr(), K, rows, K, c.data_ptr(), 260)
    ref = a.float() @ b.float().T
    torch.cuda.synchronize()
    assert torch.isnan(c[:, 256:]).all()  # nothing past the 256 columns
    assert torch.allclose(c[:, :256], ref, rtol=1e-5, atol=1e-4 * K ** 0.5), float((c[:, :256] - ref).abs().max())


@pytest.mark.parametrize("n", [128, 384, 640])
def test_gradients_of_ragged_batches(torch_cuda, n):
    torch = torch_cuda
    from tardiis_and_claritas_gb300 import lib as L
    net = L.Network(0, max_batch=1024, seed=1)
    p = M.init_params(11)
    net.set_params(p)
    rng = np.random.default_rng(n)
    x = rng.normal(size=(n, 6)).astype(np.float32)
    t = np.stack([np.sin(x[:, 0]), np.cos(x[:, 3]) * x[:, 4], 0.3 * x[:, 5] ** 2], axis=1).astype(np.float32)
    xd, td = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
    loss, g = net.gradients(xd.data_ptr(), td.data_ptr(), n)
    loss_or, g_or = M.loss_and_grad(p, x, t)
    assert abs(loss - loss_or) < 1e-3 * loss_or
    k = 0
    for li, (o, i) in enumerate(M.LAYERS):
        for name, cnt in (("W", o * i), ("b", o)):
            a, b = g[k:k + cnt].astype(np.float64), g_or[k:k + cnt]
            assert np.linalg.norm(a - b) < 2e-2 * max(np.linalg.norm(b), 1e-12), (li + 1, name)
            k += cnt
    net.close()


def test_training_steps_follow_their_inputs(torch_cuda):
    """The captured step reads its rows, weights and learning rate from device memory: calls with other index
    arrays, another row count, weights on and off and another batch equal a fresh network given the same calls."""
    torch = torch_cuda
    from tardiis_and_claritas_gb300 import lib as L
    rng = np.random.default_rng(5)
    x = torch.from_numpy(rng.normal(size=(3000, 6)).astype(np.float32)).cuda()
    t = torch.from_numpy(rng.normal(size=(3000, 3)).astype(np.float32)).cuda()
    w = torch.from_numpy(rng.uniform(0.5, 2.0, size=(3000, 3)).astype(np.float32)).cuda()
    calls = [(512, 700, False, 1e-3), (512, 2999, True, 5e-4), (256, 900, False, 1e-3), (512, 512, True, 2e-3)]
    nets = [L.Network(0, max_batch=512, seed=2) for _ in range(2)]
    for batch, rows, weighted, lr in calls:
        idx = torch.from_numpy(rng.permutation(3000)[:rows].astype(np.int32)).cuda()
        before = nets[0].get_params()
        losses = []
        for k, net in enumerate(nets):
            if k == 1:
                net.set_loss_weights(0)  # a fresh setting before every call of the second network
            net.set_loss_weights(w.data_ptr() if weighted else 0)
            losses.append(net.train(x.data_ptr(), t.data_ptr(), idx.clone().data_ptr() if k else idx.data_ptr(), rows, batch, lr))
        a, b = nets[0].get_params(), nets[1].get_params()
        assert np.abs(a - before).max() > 0.1 * lr  # the steps moved the weights
        assert abs(losses[0] - losses[1]) < 1e-4 * losses[0]
        # FP32 atomic order is the only difference between the two networks
        assert np.linalg.norm(a - b) < 1e-3 * np.linalg.norm(a - before) + 1e-7 * np.linalg.norm(a)
    for net in nets:
        net.close()


@pytest.mark.parametrize("n", [128, 640, 1024])
def test_gradients_are_the_same_bits_in_every_run(torch_cuda, n):
    """Partial sums are added in a fixed order, and those of a larger batch before leave nothing behind."""
    torch = torch_cuda
    from tardiis_and_claritas_gb300 import lib as L
    rng = np.random.default_rng(3)
    x = torch.from_numpy(rng.normal(size=(1024, 6)).astype(np.float32)).cuda()
    t = torch.from_numpy(rng.normal(size=(1024, 3)).astype(np.float32)).cuda()
    got = []
    for before in (0, 1024, n):
        net = L.Network(0, max_batch=1024, seed=1)
        net.set_params(M.init_params(11))
        if before:
            net.gradients(x.data_ptr(), t.data_ptr(), before)
        got.append(net.gradients(x.data_ptr(), t.data_ptr(), n)[1])
    np.testing.assert_array_equal(got[0], got[1])
    np.testing.assert_array_equal(got[0], got[2])
