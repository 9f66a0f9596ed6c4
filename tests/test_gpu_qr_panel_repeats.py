"""QR panels with sums pushed to every rank: the same bits from every repetition."""
import numpy as np
import pytest
import torch

import tnpy_gb300.kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("half,n", [(20, 34), (64, 128), (640, 64), (1024, 192)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_gauge_move_repeats(half, n, precision):
    rng = np.random.RandomState(half + n)
    site = torch.from_numpy(rng.standard_normal((half, 2, n))).cuda()
    nb = torch.from_numpy(rng.standard_normal((n, 2, 16))).cuda()
    first = None
    for _ in range(40):
        a, b = site.clone(), nb.clone()
        K.gauge_move(1, a, b, precision=precision)
        if first is None:
            first = a, b
        assert torch.equal(a, first[0]) and torch.equal(b, first[1])
