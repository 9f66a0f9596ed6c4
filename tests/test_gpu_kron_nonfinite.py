"""Blocks with Inf, NaN or entries beyond FP32 among the pairs of a Kronecker eigensolve: reported for the block, and the
others are as without it."""
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
    return w[None] if left else w[:, None]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf, 1e60])
@pytest.mark.parametrize("m,chi,batch", [(8, 8, 3), (20, 24, 3), (8, 8, 160)])
def test_kron_eigh_beside_a_bad_block(m, chi, batch, bad, precision):
    rng = np.random.RandomState(m)
    nodes = [(_node(rng, m, True), _node(rng, m, False)) for _ in range(batch)]
    nodes[1][0][0, 3, 2, 1] = nodes[1][0][0, 3, 1, 2] = bad
    pairs = [tuple(torch.from_numpy(w).cuda() for w in p) for p in nodes]
    ev, vec, ks, iters = T.kron_eigh(pairs, chi, torch.device("cuda"), precision=precision)
    it = iters.cpu().numpy()
    if not np.isfinite(bad):
        assert it[1] < 0  # reported as not converged
    for b in (0, 2):
        w1, w2 = nodes[b]
        h = sum(np.kron(w1[0, i], w2[i, 0]) for i in range(5))
        e = np.linalg.eigvalsh(h)
        assert it[b] > 0
        assert np.abs(ev[b, : ks[b]].cpu().numpy() - e[: ks[b]]).max() <= 4e-8 * np.abs(e).max()


