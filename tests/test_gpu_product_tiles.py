"""GPU: the plain product with 256-wide rows at the edges of its two tiles.

Up to 76 row tiles a CTA makes 128 rows of 64 columns, from there on 128 rows of all 256 columns in a ring of two
stages. Checked against a PyTorch FP32 product of the same BF16 values: only the summation order differs (1e-5
relative, 1e-4 sqrt(K) absolute for unit normals, as for the other sizes).
"""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    import torch
    from tardiis_and_claritas_gb300.build_ext import build
    build()
    return torch


# 76 tiles; 77, the last with one row, a row short, full; K of one, two, three and nine stages
@pytest.mark.parametrize("rows,K", [(9728, 128), (9729, 64), (9729, 128), (9855, 192), (9856, 576)])
def test_product_on_either_side_of_the_wide_tile(torch_cuda, rows, K):
    torch = torch_cuda
    from tardiis_and_claritas_gb300 import lib as L
    g = torch.Generator(device="cpu").manual_seed(rows + K)
    a = torch.randn(rows, K + 8, generator=g).to(torch.bfloat16).cuda()[:, :K]
    b = torch.randn(256, K, generator=g).to(torch.bfloat16).cuda()
    c = torch.full((rows + 1, 260), float("nan"), dtype=torch.float32, device="cuda")
    L.bf16_gemm_n256(a.data_ptr(), K + 8, b.data_ptr(), K, rows, K, c.data_ptr(), 260)
    ref = a.float() @ b.float().T
    torch.cuda.synchronize()
    assert torch.isnan(c[:, 256:]).all() and torch.isnan(c[rows]).all()  # nothing past the rows and columns
    assert torch.allclose(c[:rows, :256], ref, rtol=1e-5, atol=1e-4 * K ** 0.5), float((c[:rows, :256] - ref).abs().max())
