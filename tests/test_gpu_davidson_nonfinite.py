"""Operators with Inf or NaN, or that overflow on the way, end a Davidson solve with an error."""
import numpy as np
import pytest
import torch

import tnpy_gb300.kernels as K

pytestmark = pytest.mark.gpu


def _solve(a, x):
    n = a.shape[0]
    one = torch.ones((1, 1, 1), dtype=torch.float64, device="cuda")
    op = (torch.from_numpy(a).cuda().reshape(n, 1, n), one.reshape(1, 1, 1, 1), one)
    t = torch.from_numpy(x.reshape(n, 1, 1).copy()).cuda()
    return K.davidson1(*op, t, tol=1e-10, max_iter=60, max_basis=40)


@pytest.mark.parametrize("n", [1, 2, 8, 33, 50])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("where", ["last", "diagonal", "pair", "all"])
def test_bad_entries(n, bad, where):
    rng = np.random.RandomState(n)
    a = rng.standard_normal((n, n))
    a = a + a.T
    if where == "last":
        a[n - 1, n - 1] = bad
    elif where == "diagonal":
        np.fill_diagonal(a, bad)
    elif where == "pair":
        a[0, n - 1] = a[n - 1, 0] = bad
    else:
        a[:] = bad
    for x in (rng.standard_normal(n), np.eye(n)[0]):
        with pytest.raises(ValueError):
            _solve(a, x)


@pytest.mark.parametrize("n", [3, 8, 33, 50])
@pytest.mark.parametrize("sign", [1.0, -1.0, 0.0])
def test_overflow_in_a_later_product(n, sign):
    rng = np.random.RandomState(n)
    a = np.full((n, n), 1.5e308)
    a *= np.sign(rng.standard_normal((n, n))) if sign == 0.0 else sign
    a = np.triu(a) + np.triu(a, 1).T
    a[0, :] = a[:, 0] = 1e290 * rng.standard_normal(n)  # the first product, of e_0, is finite
    with pytest.raises(ValueError):
        _solve(a, np.eye(n)[0])
