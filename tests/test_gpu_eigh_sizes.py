"""Batched FP64 Jacobi at the edges of its forms (n = 64 queue, n = 112 shared memory), with block
structure, equal diagonals and mixed sizes, against numpy."""
import numpy as np
import pytest
import torch

import tnpy_gb300.kernels as K

pytestmark = pytest.mark.gpu


def _matrix(n, kind):
    rng = np.random.RandomState(n)
    a = rng.standard_normal((n, n))
    if kind == "blocks":  # a conserved label: zero between different labels
        q = rng.randint(0, 4, size=n)
        a = a * (q[:, None] == q[None, :])
    elif kind == "equal_diagonal":
        np.fill_diagonal(a, 1.5)
        a[n // 2:, :] = 0.0
        a[:, n // 2:] = 0.0
    elif kind == "zero":
        a = np.zeros((n, n))
    elif kind == "tiny":
        a = 1e-140 * a
    return a + a.T


@pytest.mark.parametrize("kind", ["dense", "blocks", "equal_diagonal", "zero", "tiny"])
@pytest.mark.parametrize("sizes", [(1, 2, 5), (63, 64, 31), (65, 66), (112, 3), (113,), (150, 64)])
def test_eigh_batched(sizes, kind):
    mats = [_matrix(n, kind) for n in sizes]
    keep = max(sizes)
    w, v = K.eigh_batched([torch.from_numpy(m).cuda() for m in mats], keep=keep)
    for i, (n, a) in enumerate(zip(sizes, mats)):
        wi, vi = w[i, :n].cpu().numpy(), v[i, :n, :n].cpu().numpy()
        # about one rounding of |a|_F per sweep and index: n * 10 sweeps
        tol = 10 * n * 2.0 ** -52
        norm = np.linalg.norm(a)
        assert np.abs(wi - np.linalg.eigvalsh(a)).max() <= tol * norm
        assert np.abs(vi.T @ vi - np.eye(n)).max() <= tol
        assert np.abs(a @ vi - vi * wi).max() <= tol * norm
        assert bool(torch.isnan(w[i, n:]).all()) and not bool(v[i, n:].any())
