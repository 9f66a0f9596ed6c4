"""One-sided Jacobi SVD of columns whose squared norms, or the products of two of them, leave the normal range of
FP64: the whole matrix scaled down, and columns graded from one to there."""
import numpy as np
import pytest
import torch

import tnpy_gb300.kernels as K

pytestmark = pytest.mark.gpu


def _check(m, n, a, scale):
    tol = 10 * m * n ** 0.5 * 2.0 ** -53  # rotations round each column about once per sweep and index
    t = torch.from_numpy(np.ascontiguousarray(a * scale)).cuda()
    ref = np.linalg.svd(a, compute_uv=False)
    _, s0, _ = K.svd(t, want_u=False, want_vt=False)
    u, s, vt = (x.cpu().numpy() for x in K.svd(t))
    s0, s = s0.cpu().numpy() / scale, s / scale
    assert np.abs(s0 - ref).max() <= tol * ref[0]
    assert np.abs(s - ref).max() <= tol * ref[0]
    assert np.abs(vt @ vt.T - np.eye(n)).max() <= 10 * n * 2.0 ** -53 * 12
    assert np.abs(u.T @ u - np.eye(n)).max() <= tol
    assert np.abs((u * s) @ vt - a).max() <= tol * ref[0]


@pytest.mark.parametrize("m,n", [(2, 2), (12, 12), (33, 5), (64, 31), (1030, 6)])
@pytest.mark.parametrize("scale", [1e-140, 1e-148, 1e-152, 1e-156, 1e-160])
def test_svd_of_a_tiny_matrix(m, n, scale):
    _check(m, n, np.random.RandomState(m + n).standard_normal((m, n)), scale)


@pytest.mark.parametrize("m,n", [(12, 12), (64, 31), (1030, 6)])
@pytest.mark.parametrize("last", [-152, -159])
def test_svd_of_columns_graded_to_tiny(m, n, last):
    a = np.random.RandomState(m + n).standard_normal((m, n))
    a[:, n // 2:] *= np.logspace(last + 8, last, n - n // 2)
    _check(m, n, a, 1.0)
