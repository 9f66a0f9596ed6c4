"""Split-BF16 GEMM by single CTAs and by CTA pairs: ragged tiles of every width, and the same bits from all of
them (each output sums the same products in the same order)."""
import pytest
import torch

import tnpy_gb300.kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(100, 100, 64), (257, 129, 70), (300, 130, 1000), (2500, 385, 130),  # pairs, 128 columns
                                   (4000, 1500, 128),  # pairs, 192 columns
                                   (3000, 3001, 200), (9728, 512, 65),  # pairs, 256 columns
                                   (127, 19399, 90)])  # single CTAs
def test_tiles_agree(m, n, k):
    g = torch.Generator(device="cuda").manual_seed(m)
    a, b = (torch.randn(s, k, generator=g, dtype=torch.float64, device="cuda") for s in (m, n))
    c, ref = K.gemm_bf16x3(a, b), a @ b.T
    # three products of splits that drop 2^-17 of an operand each; FP32 sums of 3 k terms
    assert float((c - ref).abs().max()) <= (2.0 ** -16 + 2.0 ** -22) * float((a.abs() @ b.abs().T).max())
    for i, j in ((0, 0), (max(m - 90, 0), max(n - 70, 0))):  # corner blocks as products of their own
        assert torch.equal(K.gemm_bf16x3(a[i:i + 90].contiguous(), b[j:j + 70].contiguous()), c[i:i + 90, j:j + 70])
