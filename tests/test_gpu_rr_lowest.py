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


def _form(form, n):
    rng = np.random.RandomState(n)
    if form == "diagonal":
        return np.diag(rng.permutation(np.linspace(-2.0, 3.0, n)))
    if form == "twice":  # every eigenvalue twice
        m = rng.standard_normal((n // 2, n // 2))
        return np.kron(np.eye(2), m + m.T)
    a = np.diag(np.arange(n) - 5.0)
    if form == "arrow":
        a[-1, :-1] = a[:-1, -1] = rng.standard_normal(n - 1)
    if form == "dense":
        t = rng.standard_normal((n, n))
        a = t + t.T
    if form == "weak":  # the first vector solves it to 1e-9
        t = rng.standard_normal((n - 1, n - 1))
        a[1:, 1:] += 0.1 * (t + t.T)
        a[0, 1:] = a[1:, 0] = 1e-9 * rng.standard_normal(n - 1)
        a[0, 0] = -20.0
    return a


@pytest.mark.parametrize("n", [2, 6, 18, 32, 40, 64])
@pytest.mark.parametrize("form", ["zero", "ones", "diagonal", "twice", "arrow", "dense", "weak"])
@pytest.mark.parametrize("scale", [1.0, 1e-140, 1e140])
def test_davidson_over_the_whole_space(n, form, scale):
    """A basis that grows to the whole space: projected matrices of every size up to n."""
    a = {"zero": np.zeros((n, n)), "ones": np.ones((n, n))}.get(form)
    a = scale * (_form(form, n) if a is None else a)
    w = np.linalg.eigvalsh(a)
    norm = max(abs(w[0]), abs(w[-1]))
    one = torch.ones((1, 1, 1), dtype=torch.float64, device="cuda")
    x = torch.from_numpy(np.random.RandomState(n + 1).standard_normal((n, 1, 1))).cuda()
    e, rn, its, ok = K.davidson1(torch.from_numpy(a).cuda().reshape(n, 1, n), one.reshape(1, 1, 1, 1), one, x,
                                 tol=1e-11 if scale == 1.0 else 0.0, max_iter=200, max_basis=64)
    v = x.cpu().numpy().ravel()
    assert abs(np.linalg.norm(v) - 1.0) <= 1e-13
    r = np.linalg.norm(a @ v - e * v)
    # the reported residual is the true one, and the value is its own Rayleigh quotient
    assert abs(r - rn) <= 64 * n * 2.0 ** -53 * norm
    assert abs(e - v @ a @ v) <= 64 * n * 2.0 ** -53 * norm
    if ok and scale == 1.0:  # an eigenpair; the lowest one where the start and the form let a Davidson reach it
        assert r <= 2e-11 * max(1.0, abs(e))
        gap = e - w[0] if form not in ("diagonal", "weak") else np.abs(e - w).min()
        assert gap <= 2e-11 * max(1.0, abs(e))


@pytest.mark.parametrize("n", [3, 5, 12, 24, 37, 50])
@pytest.mark.parametrize("seed", [0, 1, 2, 3])
def test_davidson_sign_is_that_of_jacobi_steps(n, seed):
    """The generalised solver with B = 1 is the same iteration with a Jacobi Rayleigh-Ritz in every step."""
    rng = np.random.RandomState(100 * n + seed)
    a = rng.standard_normal((n, n))
    a = a + a.T + np.diag(rng.uniform(-1.0, 1.0, n) * 5 * (seed % 2))
    one = torch.ones((1, 1, 1), dtype=torch.float64, device="cuda")
    op = (torch.from_numpy(a).cuda().reshape(n, 1, n), one.reshape(1, 1, 1, 1), one)
    eye = (torch.eye(n, dtype=torch.float64, device="cuda").reshape(n, 1, n), one.reshape(1, 1, 1, 1), one)
    x = torch.from_numpy(rng.standard_normal((n, 1, 1))).cuda()
    y = x.clone()
    K.davidson1(*op, x, tol=1e-9, max_iter=200, max_basis=64)
    K.gdavidson1(*op, *eye, y, tol=1e-9, max_iter=200, max_basis=64)
    assert float((x * y).sum()) > 0.9


@pytest.mark.parametrize("max_basis", [4, 7, 24])
@pytest.mark.parametrize("chi", [8, 20])
def test_davidson_sign_through_restarts(max_basis, chi):
    """Stacked chains run the same iteration, restarts included, with a Jacobi Rayleigh-Ritz in every step."""
    g = torch.Generator(device="cuda").manual_seed(chi + max_basis)
    rand = lambda *s: torch.randn(*s, generator=g, dtype=torch.float64, device="cuda")
    batch = 4
    L, R = ((e + e.transpose(1, 3)).contiguous() for e in (rand(batch, chi, 1, chi), rand(batch, chi, 1, chi)))
    w = torch.diag(torch.tensor([1.0, 0.6], dtype=torch.float64, device="cuda")).reshape(1, 1, 2, 2)
    x = rand(batch, chi, 2, chi)
    y = x.clone()
    K.batched_davidson1(L, w.expand(batch, 1, 1, 2, 2).contiguous(), R, y, tol=1e-10, max_iter=400, max_basis=max_basis)
    for i in range(batch):
        xi = x[i].clone()
        e, rn, its, ok = K.davidson1(L[i], w, R[i], xi, tol=1e-10, max_iter=400, max_basis=max_basis)
        dot = float((xi * y[i]).sum())
        if ok and abs(dot) > 0.9:
            assert dot > 0, (i, its)
