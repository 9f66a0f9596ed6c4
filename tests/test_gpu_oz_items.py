"""Ozaki GEMM with several tiles a CTA: counts around a multiple of the SMs, K blocks and chunks at their edges,
batches with a mask, split K; every tile against FP64."""
import pytest
import torch

import tnpy_gb300.kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,m,n,k,nsplit", [(1, 1, 1, 1, 1), (1, 128, 64, 32, 1), (1, 129, 65, 33, 2),
                                                (1, 2432, 512, 64, 1), (1, 2432, 513, 480, 1), (1, 2400, 1500, 481, 1),
                                                (1, 3000, 900, 961, 3), (200, 100, 64, 70, 1), (40, 130, 200, 500, 4)])
@pytest.mark.parametrize("alpha,beta", [(1.0, 0.0), (-0.5, 1.0)])
def test_every_tile(batch, m, n, k, nsplit, alpha, beta):
    g = torch.Generator(device="cuda").manual_seed(m + k)
    rand = lambda *s: torch.randn(*s, generator=g, dtype=torch.float64, device="cuda")
    a, b, c = rand(batch, m, k), rand(batch, k, n), rand(batch, m, n)
    mask = (torch.arange(batch, device="cuda") % 7 != 3) if batch > 1 else None
    out = K.gemm_oz_batched(a, b, c.clone(), alpha=alpha, beta=beta, nsplit=nsplit, mask=mask)
    ref = alpha * (a @ b) + beta * c
    if mask is not None:
        assert torch.equal(out[~mask], c[~mask])
        out, ref = out[mask], ref[mask]
    # 2^-52 of the row and column maxima a product, double-FP32 sums to 2^-46 of the running sum, chunk by chunk
    tol = 2.0 ** -46 * (2 + k / 480) * float((a.abs() @ b.abs()).max())
    tol += 2.0 ** -51 * k * float(a.abs().max() * b.abs().max()) + 2.0 ** -51 * float(ref.abs().max())
    assert float((out - ref).abs().max()) <= tol
