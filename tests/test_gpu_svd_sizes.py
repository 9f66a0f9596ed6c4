"""One-sided Jacobi SVD at odd and small sizes, on both triangles, graded, repeated and zero columns,
with and without vectors, against numpy."""
import numpy as np
import pytest
import torch

import tnpy_gb300.kernels as K

pytestmark = pytest.mark.gpu


def _matrix(m, n, kind):
    rng = np.random.RandomState(m + 3 * n)
    a = rng.standard_normal((m, n))
    if kind in ("upper", "lower"):
        a = np.triu(a) * np.logspace(0, -12, n)[:, None] if kind == "upper" else np.tril(a) * np.logspace(0, -12, n)
    elif kind == "zeros":
        a[:, ::3] = 0.0
    elif kind == "tiny":
        a *= 1e-120
    return a


@pytest.mark.parametrize("m,n,kind", [
    (1, 1, "dense"), (2, 2, "dense"), (9, 3, "dense"), (33, 33, "dense"), (130, 67, "dense"), (1030, 12, "dense"),
    (64, 64, "upper"), (64, 64, "lower"), (31, 31, "upper"), (40, 40, "zeros"), (50, 20, "zeros"), (24, 24, "tiny"),
])
def test_svd(m, n, kind):
    a = _matrix(m, n, kind)
    t = torch.from_numpy(a).cuda()
    ref = np.linalg.svd(a, compute_uv=False)
    tol = 10 * m * n ** 0.5 * 2.0 ** -53  # rotations round each column about once per sweep and index
    _, s0, _ = K.svd(t, want_u=False, want_vt=False)
    u, s, vt = (x.cpu().numpy() for x in K.svd(t))
    assert np.abs(s0.cpu().numpy() - ref).max() <= tol * ref[0]
    assert np.abs(s - ref).max() <= tol * ref[0]
    assert np.abs(vt @ vt.T - np.eye(n)).max() <= 10 * n * 2.0 ** -53 * 12
    assert np.abs((u * s) @ vt - a).max() <= tol * ref[0]
