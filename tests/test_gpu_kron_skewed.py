"""Kronecker eigensolver where the two nodes differ: both orders, at the edges of the narrow form (one node of at most
8 states beside one of more than 16) and of the sums that stop at the nodes' dimensions, against numpy."""
import numpy as np
import pytest
import torch

from tnpy_gb300 import tsdrg as T

pytestmark = pytest.mark.gpu


def _node(rng, m, left):
    sp, sz = 0.3 * rng.standard_normal((m, m)), 0.2 * rng.standard_normal((m, m))
    h, eye = np.diag(np.sort(rng.uniform(-6, 0, m))), np.eye(m)
    sz = sz + sz.T
    w = np.stack([eye, 0.5 * sp, 0.5 * sp.T, sz, h] if left else [h, sp.T, sp, sz, eye])
    return torch.from_numpy(w[None] if left else w[:, None]).cuda()


@pytest.mark.parametrize("m1,m2", [(17, 1), (1, 17), (17, 8), (8, 17), (32, 8), (8, 32), (24, 4), (4, 24), (21, 5), (31, 7),
                                   (17, 9), (9, 17), (32, 16), (24, 25), (25, 24), (25, 25)])
@pytest.mark.parametrize("chi,batch", [(4, 2), (17, 160)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_skewed_blocks(m1, m2, chi, batch, precision):
    rng = np.random.RandomState(m1 * 100 + m2)
    few = [(_node(rng, m1, True), _node(rng, m2, False)) for _ in range(2)]
    pairs = [few[b % 2] for b in range(batch)]
    ev, vec, ks, iters = T.kron_eigh(pairs, chi, torch.device("cuda"), precision=precision)
    assert int(iters.min()) > 0
    m = m1 * m2
    for b in (0, batch - 1):
        w1, w2 = (w.cpu().numpy() for w in pairs[b])
        h = sum(np.kron(w1[0, i], w2[i, 0]) for i in range(5))
        e = np.linalg.eigvalsh(h)
        scale = max(abs(e[0]), abs(e[-1]))
        v, lam = vec[b, :m, : ks[b]].cpu().numpy(), ev[b, : ks[b]].cpu().numpy()
        # FP64: residual 1e-13 of the scale a vector; otherwise 3e-6, second order in the values
        # (gaps of ~1e-2 of the scale)
        rtol, etol = (1e-13, 1e-13) if precision == "fp64" else (1e-5, 1e-8)
        assert np.abs(lam - e[: ks[b]]).max() <= 4 * etol * scale
        assert np.abs(np.linalg.norm(h @ v - v * lam, axis=0)).max() <= 4 * rtol * scale
        assert np.abs(v.T @ v - np.eye(ks[b])).max() <= m * 2.0 ** -50
