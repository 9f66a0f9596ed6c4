"""Zero matrices and operators: the lowest value is zero, with a unit vector."""
import numpy as np
import pytest
import torch

import tnpy_gb300.kernels as K

pytestmark = pytest.mark.gpu


def _zero(*s):
    return torch.zeros(s, dtype=torch.float64, device="cuda")


@pytest.mark.parametrize("n", [1, 2, 17, 32, 33, 64])
@pytest.mark.parametrize("entry", [0.0, -0.0, 1e-310])
def test_lowest_pair_of_a_zero_matrix(n, entry):
    e, v = K.eigh_batched([torch.full((n, n), entry, dtype=torch.float64, device="cuda")], keep=1)
    assert abs(float(e[0, 0])) <= 64 * 1e-310
    assert abs(float(v[0, :, 0].norm()) - 1.0) <= 1e-14


@pytest.mark.parametrize("chi", [2, 8, 20])
@pytest.mark.parametrize("batch", [1, 3])
def test_stacked_davidson_of_zero_operators(chi, batch):
    g = torch.Generator(device="cuda").manual_seed(chi)
    x = torch.randn(batch, chi, 2, chi, generator=g, dtype=torch.float64, device="cuda")
    w = torch.eye(2, dtype=torch.float64, device="cuda").reshape(1, 1, 1, 2, 2).repeat(batch, 1, 1, 1, 1)
    r = K.batched_davidson1(_zero(batch, chi, 1, chi), w, _zero(batch, chi, 1, chi), x, tol=1e-10)
    assert np.all(np.abs(torch.as_tensor(r[0]).cpu().numpy()) == 0.0)
    assert bool(((x.reshape(batch, -1).norm(dim=1) - 1.0).abs() <= 1e-12).all())


def test_generalised_davidson_of_a_zero_operator():
    n = 20
    one = torch.ones((1, 1, 1), dtype=torch.float64, device="cuda")
    eye = torch.eye(n, dtype=torch.float64, device="cuda").reshape(n, 1, n)
    x = torch.randn(n, 1, 1, dtype=torch.float64, device="cuda")
    e = K.gdavidson1(_zero(n, 1, n), one.reshape(1, 1, 1, 1), one, eye, one.reshape(1, 1, 1, 1), one, x, tol=1e-9)[0]
    assert float(e) == 0.0 and bool(torch.isfinite(x).all())
