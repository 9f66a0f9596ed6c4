"""FP64-class environment updates and gauge moves on both sides of the sizes from which the products leave
the FP64 pipe, against FP64."""
import pytest
import torch

import tnpy_gb300.kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chi_l,chi_r", [(1, 4), (16, 20), (64, 60), (100, 130), (150, 150), (150, 260), (190, 170)])
@pytest.mark.parametrize("direction", [1, -1])
def test_env_update(chi_l, chi_r, direction):
    g = torch.Generator(device="cuda").manual_seed(chi_l + chi_r)
    rand = lambda *s: torch.randn(*s, generator=g, dtype=torch.float64, device="cuda")
    c = chi_l if direction == 1 else chi_r
    e, a, w = rand(c, 5, c), rand(chi_l, 2, chi_r), rand(5, 5, 2, 2)
    out, ref = (K.env_update(direction, e, a, w, precision=p) for p in ("mixed", "fp64"))
    mag = K.env_update(direction, e.abs(), a.abs(), w.abs(), precision="fp64")
    # two products of ~2^-47 an operation, whose errors add like a random walk at the most
    assert float(((out - ref).abs() / mag).max()) <= 2.0 ** -43


@pytest.mark.parametrize("chi_l,chi_r", [(20, 36), (80, 90), (130, 120), (170, 150)])
def test_gauge_move(chi_l, chi_r):
    g = torch.Generator(device="cuda").manual_seed(chi_l)
    rand = lambda *s: torch.randn(*s, generator=g, dtype=torch.float64, device="cuda")
    s, nb = rand(chi_l, 2, chi_r), rand(chi_r, 2, 50)
    got, want = [], []
    for p, out in (("mixed", got), ("fp64", want)):
        a, b = s.clone(), nb.clone()
        K.gauge_move(1, a, b, precision=p)
        out += [a, b]
    for x, y in zip(got, want):  # random matrices: condition of a few hundred
        assert float((x - y).abs().max()) <= 2.0 ** -47 * 64 * chi_r ** 0.5 * 300 * float(y.abs().max())
