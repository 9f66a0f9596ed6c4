"""Shared-memory QR (single sites and stacked chains) at odd, square, tall and largest shapes, zero and
badly scaled columns, against the defining properties and LAPACK's sign convention."""
import numpy as np
import pytest
import torch

import tnpy_gb300.kernels as K

pytestmark = pytest.mark.gpu


def _check(m, q, r):
    n = m.shape[1]
    tol = 20 * m.shape[0] * 2.0 ** -53  # Householder: a few m u, columnwise
    assert np.abs(q.T @ q - np.eye(n)).max() <= tol
    assert np.all(np.tril(r, -1) == 0.0)
    col = np.linalg.norm(m, axis=0)
    assert np.all(np.linalg.norm(q @ r - m, axis=0) <= tol * col + 1e-300)


@pytest.mark.parametrize("m,n", [(1, 1), (2, 1), (5, 5), (7, 3), (31, 16), (32, 32), (64, 32), (129, 31), (256, 17)])
@pytest.mark.parametrize("kind", ["normal", "zero_columns", "scaled"])
def test_qr_small(m, n, kind):
    a = np.random.RandomState(m + n).standard_normal((m, n))
    if kind == "zero_columns":
        a[:, ::2] = 0.0
    elif kind == "scaled":
        a *= np.logspace(-200, 120, n)
    q, r = (t.cpu().numpy() for t in K.qr(torch.from_numpy(a).cuda()))
    _check(a, q, r)
    if kind == "normal":  # the same reflectors as LAPACK's: the same signs
        assert np.all(np.sign(np.diag(r)) == np.sign(np.diag(np.linalg.qr(a)[1])))


@pytest.mark.parametrize("batch,cl,cr", [(3, 13, 26), (1, 64, 100), (5, 50, 100), (2, 6400, 1), (80, 20, 33), (2, 56, 112)])
@pytest.mark.parametrize("direction", [1, -1])
def test_batched_gauge_move_shapes(batch, cl, cr, direction):
    g = torch.Generator(device="cuda").manual_seed(cl)
    rand = lambda *s: torch.randn(*s, generator=g, dtype=torch.float64, device="cuda")
    site = rand(batch, cl, 2, cr) if direction == 1 else rand(batch, cr, 2, cl)
    nb = rand(batch, cr, 2, 3) if direction == 1 else rand(batch, 3, 2, cr)
    a, b = site.clone(), nb.clone()
    K.batched_gauge_move(direction, a, b)
    for i in range(batch):
        if direction == 1:
            m0, q, n0, n1 = site[i].reshape(-1, cr), a[i].reshape(-1, cr), nb[i].reshape(cr, -1), b[i].reshape(cr, -1)
        else:
            m0, q = site[i].reshape(cr, -1).T, a[i].reshape(cr, -1).T
            n0, n1 = nb[i].reshape(-1, cr).T, b[i].reshape(-1, cr).T
        r = (q.T @ m0).triu().cpu().numpy()
        _check(m0.cpu().numpy(), q.cpu().numpy(), r)
        tol = 60 * m0.shape[0] * 2.0 ** -53
        assert float((n1 - torch.from_numpy(r).cuda() @ n0).abs().max()) <= tol * float(m0.norm() * n0.norm())
