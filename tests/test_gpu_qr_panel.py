"""Double-FP32 QR panels at edges of their row split: fewer rows than CTAs, ragged rows, a last panel of one
column, and heights on both sides of the one where sums are no longer pushed to every rank."""
import numpy as np
import pytest
import torch

import tnpy_gb300.kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("half,n", [(20, 34), (17, 34), (50, 64), (33, 66), (129, 65), (640, 64), (1001, 129),
                                    (3190, 34), (3300, 36), (3400, 34)])
@pytest.mark.parametrize("graded", [False, True])
def test_gauge_move_with_double_fp32_panels(half, n, graded):
    m = 2 * half
    a = np.random.RandomState(m + n).standard_normal((m, n))
    if graded:
        a *= np.logspace(0, -9, n)
    site, nb = torch.from_numpy(a.reshape(half, 2, n)).cuda(), torch.zeros((n, 2, n), dtype=torch.float64, device="cuda")
    nb[:, 0, :] = torch.eye(n)
    K.gauge_move(1, site, nb, precision="mixed")
    q, r = site.reshape(m, n).cpu().numpy(), nb[:, 0, :].cpu().numpy()
    # ~2^-47 an operation; sums of m terms grow like a random walk, 4 for the several passes, 16 for the worst entry
    tol = 64 * np.sqrt(m) * 2.0 ** -47
    assert np.abs(q.T @ q - np.eye(n)).max() <= tol
    assert np.all(np.linalg.norm(q @ r - a, axis=0) <= tol * np.linalg.norm(a, axis=0))
    rl = np.linalg.qr(a)[1]
    assert np.all(np.sign(np.diag(r)) == np.sign(np.diag(rl)))
    assert np.abs(np.tril(r, -1)).max() <= tol * np.abs(r).max()


@pytest.mark.parametrize("m,n", [(34, 34), (257, 20), (300, 64), (130, 129), (1000, 65), (2050, 97), (6400, 34), (6890, 33)])
@pytest.mark.parametrize("kind", ["normal", "zero_columns", "graded"])
def test_qr_with_fp64_panels(m, n, kind):
    a = np.random.RandomState(m + n).standard_normal((m, n))
    if kind == "zero_columns":
        a[:, ::3] = 0.0
    elif kind == "graded":
        a *= np.logspace(0, -140, n)
    q, r = (t.cpu().numpy() for t in K.qr(torch.from_numpy(a).cuda()))
    tol = 20 * m * 2.0 ** -53  # Householder: a few m u, columnwise
    assert np.abs(q.T @ q - np.eye(n)).max() <= tol
    assert np.all(np.tril(r, -1) == 0.0)
    assert np.all(np.linalg.norm(q @ r - a, axis=0) <= tol * np.linalg.norm(a, axis=0) + 1e-300)
    if kind == "normal":
        assert np.all(np.sign(np.diag(r)) == np.sign(np.diag(np.linalg.qr(a)[1])))
