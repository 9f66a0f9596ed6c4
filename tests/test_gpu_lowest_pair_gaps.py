"""Lowest pair of small matrices whose second eigenvalue lies close by (Rayleigh-Ritz kernel)."""
import numpy as np
import pytest
import torch

import tnpy_gb300.kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 8, 24, 33, 64])
@pytest.mark.parametrize("gap", [1e-1, 1e-2, 1e-3])
def test_lowest_pair_with_a_close_second(n, gap):
    for seed in range(12):
        rng = np.random.RandomState(1000 * n + seed)
        q, _ = np.linalg.qr(rng.standard_normal((n, n)))
        w = np.concatenate([[-1.0, -1.0 + gap], rng.uniform(-1.0 + 2.0 * gap, 1.0, n - 2)])
        a = (q * w) @ q.T
        a = 0.5 * (a + a.T)
        e, v = K.eigh_batched([torch.from_numpy(a).cuda()], keep=1)
        e, v = float(e[0, 0]), v[0, :, 0].cpu().numpy()
        # an eigenvector to rounding: the product's and its own, n terms each (the bounds of test_gpu_rr_lowest.py)
        assert abs(e - np.linalg.eigvalsh(a)[0]) <= 8 * n * 2.0 ** -53
        assert np.linalg.norm(a @ v - e * v) <= 16 * n * 2.0 ** -53
        assert abs(np.linalg.norm(v) - 1.0) <= 8 * n * 2.0 ** -53
