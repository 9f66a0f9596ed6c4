"""Lowest pair of small symmetric matrices far from unit scale, and of ones that hold Inf or NaN."""
import numpy as np
import pytest
import torch

import tnpy_gb300.kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 5, 24, 33, 64])
@pytest.mark.parametrize("scale", [1e-290, 1e-160, 1e-38, 1e-26, 1e-24, 1e-18, 1e18, 1e26, 1e38, 1e160, 1e290])
def test_lowest_pair_at_scale(n, scale):
    a = np.random.RandomState(n).standard_normal((n, n))
    a = a + a.T
    w = np.linalg.eigvalsh(a)
    e, v = K.eigh_batched([torch.from_numpy(a * scale).cuda()], keep=1)
    e, v = float(e[0, 0]) / scale, v[0, :, 0].cpu().numpy()
    norm = np.linalg.norm(a, 2)
    assert abs(e - w[0]) <= 8 * n * 2.0 ** -53 * norm
    assert abs(np.linalg.norm(v) - 1.0) <= 8 * n * 2.0 ** -53
    assert np.linalg.norm(a @ v - e * v) <= 16 * n * 2.0 ** -53 * norm


@pytest.mark.parametrize("n", [1, 5, 33, 64])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_lowest_pair_of_a_non_finite_matrix(n, bad):
    a = np.random.RandomState(n).standard_normal((n, n))
    a = a + a.T
    a[n // 2, n - 1] = a[n - 1, n // 2] = bad
    e, v = K.eigh_batched([torch.from_numpy(a).cuda()], keep=1)
    assert not bool(torch.isfinite(e).all())
