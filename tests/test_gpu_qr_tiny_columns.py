"""Shared-memory QR of columns whose norm is subnormal, or becomes so after the reflectors before."""
import numpy as np
import pytest
import torch

import tnpy_gb300.kernels as K

pytestmark = pytest.mark.gpu


def _columns(m, n, kind):
    a = np.random.RandomState(m + n).standard_normal((m, n))
    if kind == "subnormal":
        return a * 4e-310
    if kind == "graded":  # normal to subnormal, down to a few units of the last place
        return a * np.logspace(-295, -322, n)
    a[:, 1:] = a[:, :1] * np.linspace(-2.0, 2.0, n - 1)  # parallel: the remainders are rounding errors
    return a * 1e-300


@pytest.mark.parametrize("m,n", [(3, 1), (6, 3), (64, 32), (129, 31), (256, 5)])
@pytest.mark.parametrize("kind", ["subnormal", "graded", "parallel"])
@pytest.mark.parametrize("call", ["qr", "stack"])
def test_tiny_columns(m, n, kind, call):
    a = _columns(m, n, kind)
    if call == "qr":
        q, r = (t.cpu().numpy() for t in K.qr(torch.from_numpy(a).cuda()))
    else:
        site = torch.from_numpy(a.reshape(1, m, 1, n).copy()).cuda()
        nb = torch.eye(n, dtype=torch.float64, device="cuda").reshape(1, n, 1, n).contiguous()
        K.batched_gauge_move(1, site, nb)
        q, r = site.reshape(m, n).cpu().numpy(), nb.reshape(n, n).cpu().numpy()
    tol = 20 * m * 2.0 ** -53  # Householder: a few m u, columnwise
    assert np.abs(q.T @ q - np.eye(n)).max() <= tol
    # n reflectors, each with a product of m terms rounded to multiples of 2^-1074
    steps = 2 * n * m * 2.0 ** -1074
    norm = np.array([np.sqrt(((a[:, j] * 2.0 ** 900) ** 2).sum()) for j in range(n)]) * 2.0 ** -900
    assert np.all(np.abs(q @ r - a).max(axis=0) <= tol * norm + steps)
