"""Kronecker eigensolver with Hamiltonians far from unit scale: the same digits as at unit scale."""
import numpy as np
import pytest
import torch

from tnpy_gb300 import tsdrg as T

pytestmark = pytest.mark.gpu


def _node(rng, m, left, scale):
    sp, sz = 0.3 * rng.standard_normal((m, m)), 0.2 * rng.standard_normal((m, m))
    h, eye = np.diag(np.sort(rng.uniform(-6, 0, m))), np.eye(m)
    sz = sz + sz.T
    w = np.stack([eye, 0.5 * scale * sp, 0.5 * scale * sp.T, scale * sz, scale * h] if left
                 else [scale * h, sp.T, sp, sz, eye])
    return torch.from_numpy(w[None] if left else w[:, None]).cuda()


@pytest.mark.parametrize("m1,m2,chi", [(16, 16, 16), (17, 9, 32), (7, 30, 5)])
@pytest.mark.parametrize("scale", [1e-200, 1e-60, 1e-25, 1e-20, 1e-16, 1e16, 1e20, 1e60, 1e200])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_kron_eigh_at_scale(m1, m2, chi, scale, precision):
    rng = np.random.RandomState(m1 * 100 + m2)
    state = rng.get_state()
    pairs = [(_node(rng, m1, True, scale), _node(rng, m2, False, scale)) for _ in range(2)]
    rng.set_state(state)
    unit = [(_node(rng, m1, True, 1.0), _node(rng, m2, False, 1.0)) for _ in range(2)]
    ev, vec, ks, iters = T.kron_eigh(pairs, chi, torch.device("cuda"), precision=precision)
    assert int(iters.min()) > 0
    for b in range(2):
        w1, w2 = (w.cpu().numpy() for w in unit[b])
        h = sum(np.kron(w1[0, i], w2[i, 0]) for i in range(5))
        e = np.linalg.eigvalsh(h)
        norm = max(abs(e[0]), abs(e[-1]))
        v, lam = vec[b, : m1 * m2].cpu().numpy(), ev[b].cpu().numpy() / scale
        # FP64: residual 1e-13 of the scale a vector; otherwise 3e-6, second order in the values
        # (gaps of ~1e-2 of the scale)
        rtol, etol = (1e-13, 1e-13) if precision == "fp64" else (1e-5, 1e-8)
        assert np.abs(lam - e[: ks[b]]).max() <= 4 * etol * norm
        assert np.abs(np.linalg.norm(h @ v - v * lam, axis=0)).max() <= 4 * rtol * norm
        assert np.abs(v.T @ v - np.eye(ks[b])).max() <= m1 * m2 * 2.0 ** -50
