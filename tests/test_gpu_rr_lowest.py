"""Lowest pair of small symmetric matrices (Rayleigh-Ritz kernel) at odd, tiny and largest sizes."""
import numpy as np
import pytest
import torch

import tnpy_gb300.kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 7, 16, 17, 31, 32, 33, 63, 64])
@pytest.mark.parametrize("scale", [1.0, 1e-12, 1e12])
def test_lowest_pair(n, scale):
    rng = np.random.RandomState(n)
    a = rng.standard_normal((n, n))
    a = scale * (a + a.T + np.diag(np.linspace(-3.0, 5.0, n)))
    w = np.linalg.eigvalsh(a)
    e, v = K.eigh_batched([torch.from_numpy(a).cuda()], keep=1)
    e, v = float(e[0, 0]), v[0, :, 0].cpu().numpy()
    norm = np.linalg.norm(a, 2)
    assert abs(e - w[0]) <= 8 * n * 2.0 ** -53 * norm
    assert abs(np.linalg.norm(v) - 1.0) <= 8 * n * 2.0 ** -53
    assert np.linalg.norm(a @ v - e * v) <= 16 * n * 2.0 ** -53 * norm
