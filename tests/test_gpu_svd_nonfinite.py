"""Singular values of a matrix that holds Inf or NaN: not finite, or an error, and the process goes on."""
import numpy as np
import pytest
import torch

import tnpy_gb300.kernels as K
from tnpy_gb300._lib import NotConverged

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("m,n", [(1, 1), (5, 5), (40, 17), (300, 64)])
@pytest.mark.parametrize("vectors", [False, True])
def test_svd_of_a_matrix_with_a_bad_entry(m, n, bad, vectors):
    a = np.random.RandomState(m + n).standard_normal((m, n))
    a[m // 2, n // 2] = bad
    try:
        _, s, _ = K.svd(torch.from_numpy(a).cuda(), want_u=vectors, want_vt=vectors)
        assert not bool(torch.isfinite(s).all())
    except NotConverged:
        pass
    b = np.random.RandomState(m).standard_normal((m, n))
    _, s, _ = K.svd(torch.from_numpy(b).cuda(), want_u=vectors, want_vt=vectors)
    ref = np.linalg.svd(b, compute_uv=False)
    assert np.abs(s.cpu().numpy() - ref).max() <= 10 * m * n ** 0.5 * 2.0 ** -53 * ref[0]
