"""Operand preparation of the tensor-core products: Ozaki slices of rows with extreme values, both
unit-stride directions and ragged K; split-BF16 operands at rounding ties and range ends."""
import numpy as np
import pytest
import torch

import tnpy_gb300.kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("trans_a,trans_b", [(False, False), (True, False), (False, True), (True, True)])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (33, 65, 31), (130, 64, 257), (64, 129, 480)])
def test_oz_slices_exact_on_wide_rows(m, n, k, trans_a, trans_b):
    rng = np.random.RandomState(m + n + k)
    # one entry per product row: C_ij = a_ip b_pj is exact in FP64 up to one rounding, and every digit
    # of a full 53-bit significand matters
    a, b = np.zeros((m, k)), np.zeros((k, n))
    a[:, k // 2] = rng.uniform(-1, 1, m) * 2.0 ** rng.randint(-300, 300, m)
    b[k // 2] = rng.uniform(-1, 1, n) * 2.0 ** rng.randint(-300, 300, n)
    a[0, k // 2] = np.nextafter(1.0, 0.0)  # the largest digits
    b[k // 2, 0] = -np.nextafter(1.0, 0.0)
    ta = torch.from_numpy(np.ascontiguousarray(a.T if trans_a else a)).cuda()
    tb = torch.from_numpy(np.ascontiguousarray(b.T if trans_b else b)).cuda()
    c = K.gemm_oz(ta, tb, trans_a=trans_a, trans_b=trans_b).cpu().numpy()
    ref = np.outer(a[:, k // 2], b[k // 2])
    # 2^-52 of the row and column maxima dropped, and the double-FP32 sum's 2^-46
    assert np.all(np.abs(c - ref) <= 2.0 ** -45 * np.abs(ref))


def test_bf16_split_ties_and_ends():
    base = np.array([1.0, 1.5, 1.9921875, 3.0e-30, 7.0e30])
    ulp = np.array([2.0 ** -8, 2.0 ** -8 + 2.0 ** -40, 2.0 ** -8 - 2.0 ** -40, 3 * 2.0 ** -9, 2.0 ** -50])
    v = np.concatenate([(base[:, None] * (1.0 + s * ulp)).ravel() for s in (1, -1)] + [base, [0.0, 2.0 ** -120]])
    v = np.concatenate([v, -v])
    a = torch.from_numpy(np.ascontiguousarray(np.tile(v, (16, 1)).T)).cuda()  # m x 16, one value a row
    eye = torch.eye(16, dtype=torch.float64, device="cuda")
    c = K.gemm_bf16x3(a, eye).cpu().numpy()  # hi * 1 + lo * 1 in FP32
    t = torch.from_numpy(v)
    hi = t.to(torch.float32)
    # RN of an FP64 value to BF16 through FP32 with a sticky bit (round to odd)
    odd = torch.from_numpy(np.where(hi.double().numpy() == v, 0, 1))
    down = torch.where(hi.double().abs() > t.abs(), torch.nextafter(hi, torch.zeros_like(hi)), hi)
    sticky = (down.view(torch.int32) | odd.to(torch.int32)).view(torch.float32)
    h = sticky.to(torch.bfloat16).double()
    rest = t - h
    r32 = rest.to(torch.float32)
    oddr = torch.from_numpy(np.where(r32.double().numpy() == rest.numpy(), 0, 1))
    downr = torch.where(r32.double().abs() > rest.abs(), torch.nextafter(r32, torch.zeros_like(r32)), r32)
    l = (downr.view(torch.int32) | oddr.to(torch.int32)).view(torch.float32).to(torch.bfloat16).double()
    ref = (h + l).to(torch.float32).double().numpy()
    assert np.array_equal(c, np.tile(ref, (16, 1)).T)
