"""MPO step with skipped zero coefficients: partial warps and row ends of the fibres, dense and sparse
W up to the bond limit, Inf through a zero coefficient, stacked chains; against torch."""
import pytest
import torch

import tnpy_gb300.kernels as K

pytestmark = pytest.mark.gpu


def _operands(chi_l, chi_r, dl, dr, d, density, lead=()):
    g = torch.Generator(device="cuda").manual_seed(chi_l * 1000 + chi_r + dl)
    rand = lambda *s: torch.randn(*lead, *s, generator=g, dtype=torch.float64, device="cuda")
    w = rand(dl, dr, d, d)
    w = w * (torch.rand(w.shape, generator=g, dtype=torch.float64, device="cuda") < density)
    return rand(chi_l, dl, chi_l), w.contiguous(), rand(chi_r, dr, chi_r), rand(chi_l, d, chi_r)


@pytest.mark.parametrize("chi_l,chi_r,dl,dr,d,density", [
    (1, 1, 1, 1, 2, 1.0), (3, 7, 5, 5, 2, 0.15), (33, 31, 5, 6, 2, 0.15), (40, 65, 25, 25, 2, 0.05),
    (5, 9, 32, 32, 2, 1.0), (9, 5, 4, 21, 3, 0.3), (70, 129, 5, 5, 2, 0.0), (64, 64, 5, 1, 2, 1.0),
])
@pytest.mark.parametrize("lead", [(), (3,)])
def test_wcontract_left_and_right(chi_l, chi_r, dl, dr, d, density, lead):
    L, w, R, a = _operands(chi_l, chi_r, dl, dr, d, density, lead)
    for direction, E in ((1, L), (-1, R)):
        out = (K.batched_env_update if lead else K.env_update)(direction, E, a, w)
        if direction == 1:
            eq = "...awb,...asc,...wvst,...btd->...cvd"
        else:
            eq = "...cvd,...asc,...wvst,...btd->...awb"
        ref = torch.einsum(eq, E, a, w, a)
        mag = torch.einsum(eq, E.abs(), a.abs(), w.abs(), a.abs())
        terms = chi_l + chi_r * d + dl * d + dr * d
        assert bool(((out - ref).abs() <= 4 * terms * 2.0 ** -53 * mag).all())


def test_wcontract_inf_meets_zero_coefficient():
    # 0 * Inf is NaN in the dense sum: the output of a zero W is NaN where its inputs hold Inf
    L, w, R, x = _operands(8, 40, 5, 5, 2, 0.0)
    x[2, 1, 33] = float("inf")
    y = K.matvec1(L, w, R, x)
    assert bool(torch.isnan(y).all())
