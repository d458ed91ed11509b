"""GPU: the fused inference kernel at the edges of its tiles and of its persistent walk.

A CTA takes 128-row tiles, one per SM and then the next: row counts around a tile, around one tile per SM (152) and
with several tiles per CTA are checked against the numpy oracle that rounds to BF16 at the same places (2e-2 of the
largest output, the bound of the other forward tests). A row's result depends on nothing but the row: the same
inputs give the same bits wherever they stand, and nothing is written past the last row.
"""
from __future__ import annotations

import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), "..", "oracle"))
import mlp_reference as M  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 127, 128, 129, 401, 152 * 128, 152 * 128 + 1, 3 * 152 * 128 + 77])
def test_forward_at_tile_edges(n):
    import torch
    from tardiis_and_claritas_gb300 import lib as L
    from tardiis_and_claritas_gb300.build_ext import build
    build()
    net = L.Network(0, max_batch=128, seed=1)
    p = M.init_params(21)
    net.set_params(p)
    x = np.random.default_rng(n).normal(size=(n, 6)).astype(np.float32)
    x[-1] = x[0]
    xd = torch.from_numpy(x).cuda()
    y = torch.full((n + 2, 3), float("nan"), dtype=torch.float32, device="cuda")
    net.forward(xd.data_ptr(), n, y.data_ptr())
    got = y.cpu().numpy()
    assert np.isnan(got[n:]).all()
    got = got[:n]
    np.testing.assert_array_equal(got[-1], got[0])
    pick = np.unique(np.concatenate([np.arange(min(n, 300)), np.arange(max(0, n - 300), n)]))
    ref, _ = M.forward(p, x[pick])
    assert np.abs(got[pick] - ref).max() < 2e-2 * max(1.0, np.abs(ref).max())
    # the same rows in another order, and a second call
    perm = np.random.default_rng(3).permutation(n)
    y2 = torch.empty((n, 3), dtype=torch.float32, device="cuda")
    xp = torch.from_numpy(np.ascontiguousarray(x[perm])).cuda()
    net.forward(xp.data_ptr(), n, y2.data_ptr())
    np.testing.assert_array_equal(y2.cpu().numpy(), got[perm])
    net.close()
