"""Davidson on both sides of the one-cluster size limit (16384 elements), tiny and odd sites, restarts,
a start vector that is the answer, and a zero one."""
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


@pytest.mark.parametrize("chi_l,chi_r", [(2, 1), (3, 5), (10, 11), (64, 127), (64, 128), (64, 129), (100, 90)])
@pytest.mark.parametrize("max_basis,precision", [(24, "fp64"), (4, "fp64"), (24, "mixed")])
def test_davidson_residual_and_value(chi_l, chi_r, max_basis, precision):
    L, w, R, x = _operator(chi_l, chi_r)
    tol = 1e-9
    e, rn, its, ok = K.davidson1(L, w, R, x, tol=tol, max_iter=2000, max_basis=max_basis, precision=precision)
    assert ok
    limit = tol if precision == "fp64" else 2e-7
    y = K.matvec1(L, w, R, x)
    assert float((y - e * x).norm()) <= 1.01 * limit * max(1.0, abs(e)) + 1e-12
    assert abs(float(x.norm()) - 1.0) <= 1e-12
    if x.numel() <= 300:
        h = K.full_matrix1(L, w, R).cpu().numpy()
        # the value is second order in the residual over the gap
        ref = np.linalg.eigvalsh(0.5 * (h + h.T))
        assert abs(e - ref[0]) <= (2 * limit * abs(e)) ** 2 / (ref[1] - ref[0]) + 1e-12 * abs(e)


def test_davidson_from_the_answer_and_from_zero():
    L, w, R, x = _operator(10, 11)
    h = K.full_matrix1(L, w, R).cpu().numpy()
    val, vec = np.linalg.eigh(0.5 * (h + h.T))
    x = torch.from_numpy(vec[:, 0].copy()).cuda().reshape(10, 2, 11).contiguous()
    e, rn, its, ok = K.davidson1(L, w, R, x, tol=1e-30, max_iter=100)  # directions vanish at rounding level
    assert abs(e - val[0]) <= 1e-12 * abs(val[0]) and rn <= 1e-11
    with pytest.raises(ValueError):
        K.davidson1(L, w, R, torch.zeros_like(x), tol=1e-8)
