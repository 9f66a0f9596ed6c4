"""FP64 GEMM at the edges of its tiles and K splits, against torch, within the FMA chain's bound."""
import pytest
import torch

from tnpy_gb300._lib import check, lib, ptr, stream_ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ta,tb", [(0, 0), (1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("m,n,k,batch", [
    (1, 1, 1, 1), (15, 17, 16, 1), (16, 16, 129, 1), (33, 31, 15, 3), (64, 32, 160, 1), (201, 168, 840, 1),
    (65, 63, 2000, 1), (37, 500, 7, 70), (640, 700, 96, 1),
])
def test_gemm_f64_tiles_and_splits(m, n, k, batch, ta, tb):
    g = torch.Generator(device="cuda").manual_seed(m + 7 * n + 31 * k)
    rand = lambda *s: torch.randn(*s, generator=g, dtype=torch.float64, device="cuda")
    a, b = rand(batch, *((k, m + 3) if ta else (m, k + 3))), rand(batch, *((n, k + 1) if tb else (k, n + 1)))
    c0 = rand(batch, m, n + 5)
    opa = a[:, :, :m].mT if ta else a[:, :, :k]
    opb = b[:, :, :k].mT if tb else b[:, :, :n]
    for alpha, beta in ((1.0, 0.0), (-0.5, 1.5)):
        c = c0.clone()
        check("tnx_gemm_f64", lib.tnx_gemm_f64(
            ta, tb, m, n, k, alpha, ptr(a), a.shape[2], a[0].numel(), ptr(b), b.shape[2], b[0].numel(), beta, ptr(c),
            c.shape[2], c[0].numel(), batch, stream_ptr()))
        ref = alpha * (opa @ opb) + beta * c0[:, :, :n]
        # both sums round at most once per term: k + 3 roundings each of |alpha| |a| |b| + |beta c|
        bound = 2 * (k + 3) * 2.0 ** -53 * (abs(alpha) * (opa.abs() @ opb.abs()) + abs(beta) * c0[:, :, :n].abs())
        assert bool(((c[:, :, :n] - ref).abs() <= bound).all())
        assert torch.equal(c[:, :, n:], c0[:, :, n:])  # columns beyond n stay untouched
