"""Residual target of the mixed Davidson on both sides of 8192 elements, and the sign of a Ritz vector through
restarts, with the number of solves compared."""
import numpy as np
import pytest
import torch

import tnpy_gb300.kernels as K
from tnpy_gb300.model import XXZ

pytestmark = pytest.mark.gpu


def _operator(chi_l, chi_r):
    rng = np.random.RandomState(chi_l + 7 * chi_r)

    def block(chi, left):
        sp, sz, h = (0.3 * rng.standard_normal((chi, chi)) / np.sqrt(chi) for _ in range(3))
        h = h + h.T + np.diag(np.sort(rng.uniform(-8, -2, chi)))
        ops = [np.eye(chi), -0.5 * sp, -0.5 * sp.T, 0.5 * (sz + sz.T), h] if left else [h, sp.T, sp, sz + sz.T, np.eye(chi)]
        return torch.from_numpy(np.ascontiguousarray(np.stack(ops, 1))).cuda()

    w = torch.from_numpy(np.ascontiguousarray(XXZ(4, -0.5).mpo[1])).to("cuda", torch.float64)
    return block(chi_l, True), w, block(chi_r, False), torch.from_numpy(rng.standard_normal((chi_l, 2, chi_r))).cuda()


@pytest.mark.parametrize("chi_l,chi_r", [(16, 16), (16, 40), (32, 32), (64, 64), (64, 65), (91, 45), (128, 64)])
@pytest.mark.parametrize("max_basis", [6, 24])
def test_mixed_residual_target(chi_l, chi_r, max_basis):
    L, w, R, x = _operator(chi_l, chi_r)
    e, rn, its, ok = K.davidson1(L, w, R, x, tol=1e-9, max_iter=2000, max_basis=max_basis, precision="mixed")
    assert ok
    limit = 5e-8 if x.numel() <= 8192 else 2e-7
    y = K.matvec1(L, w, R, x)
    # the reported residual comes from an FP64-class product: 1 % and a few units of its rounding
    assert float((y - e * x).norm()) <= 1.01 * limit * max(1.0, abs(e)) + 1e-12
    assert rn <= limit * max(1.0, abs(e))
    assert abs(float(x.norm()) - 1.0) <= 1e-12


def test_sign_through_restarts_is_compared():
    """Stacked chains run the same iteration with a Jacobi Rayleigh-Ritz in every step."""
    compared = 0
    for max_basis, chi in [(4, 8), (7, 8), (24, 8), (4, 20), (7, 20), (24, 20)]:
        g = torch.Generator(device="cuda").manual_seed(chi + max_basis)
        rand = lambda *s: torch.randn(*s, generator=g, dtype=torch.float64, device="cuda")
        batch = 4
        L, R = ((e + e.transpose(1, 3)).contiguous() for e in (rand(batch, chi, 1, chi), rand(batch, chi, 1, chi)))
        w = torch.diag(torch.tensor([1.0, 0.6], dtype=torch.float64, device="cuda")).reshape(1, 1, 2, 2)
        x = rand(batch, chi, 2, chi)
        y = x.clone()
        K.batched_davidson1(L, w.expand(batch, 1, 1, 2, 2).contiguous(), R, y, tol=1e-10, max_iter=400, max_basis=max_basis)
        for i in range(batch):
            xi = x[i].clone()
            e, rn, its, ok = K.davidson1(L[i], w, R[i], xi, tol=1e-10, max_iter=400, max_basis=max_basis)
            dot = float((xi * y[i]).sum())
            if ok and abs(dot) > 0.9:
                assert dot > 0, (max_basis, chi, i, its)
                compared += 1
    assert compared >= 12, compared  # half of the solves at the least
