"""Not-a-number operands of the split products, with and without the sign bit
set, in every position and on both sides of the size up to which maxima and
digits are formed in one pass (512 of K): the rows or columns they stand in
must not come out as ordinary numbers, and the others must not change.

With A in [1/2, 1] the digits of a NaN alone give at least 2^1022.
"""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
NANS = {"nan": 0x7FF8000000000000, "-nan": -0x8000000000000, "-nan all ones": -1}


def cm(X):
    return X.t().contiguous().t()


def ordinary(X):
    v = torch.view_as_real(X) if X.is_complex() else X.unsqueeze(-1)
    return (v.isfinite() & (v.abs() < 1e300)).all(-1)


@pytest.mark.parametrize("bits", sorted(NANS))
@pytest.mark.parametrize("dt", [torch.float64, torch.complex128], ids=["f64", "c64"])
@pytest.mark.parametrize("K", [100, 200, 400, 512, 513, 1500])
@pytest.mark.parametrize("op", ["N", "C"])
def test_nan_rows_and_columns(mak, cuda, bits, dt, K, op):
    gen = torch.Generator(device=cuda).manual_seed(K)
    M, N = 300, 260
    A = (0.5 + 0.5 * torch.rand((M, K), generator=gen, device=cuda, dtype=torch.float64)).to(dt)
    B = (0.5 + 0.5 * torch.rand((K, N), generator=gen, device=cuda, dtype=torch.float64)).to(dt)
    nan = torch.tensor([NANS[bits]], dtype=torch.int64, device=cuda).view(torch.float64)

    def gemm(A, B):
        o = (lambda X: cm(X.mH.resolve_conj())) if op == "C" else cm
        return mak.gemm(o(A), o(B), op, op, precision="mixed")

    ref = gemm(A, B)

    def planted(X, i, j):
        X = X.clone()
        v = torch.view_as_real(X) if X.is_complex() else X.unsqueeze(-1)
        v.view(torch.int64)[i, j, 0] = nan.view(torch.int64)[0]
        return X

    C = gemm(A, planted(B, 5, 7))
    assert not ordinary(C)[:, 7].any()
    keep = [j for j in range(N) if j != 7]
    assert torch.equal(C[:, keep], ref[:, keep])
    C = gemm(planted(A, 9, 3), B)
    assert not ordinary(C)[9].any()
    keep = [i for i in range(M) if i != 9]
    assert torch.equal(C[keep], ref[keep])


@pytest.mark.parametrize("dt", [torch.float64, torch.complex128], ids=["f64", "c64"])
def test_polar_of_a_matrix_with_nan(mak, cuda, dt):
    gen = torch.Generator(device=cuda).manual_seed(11)
    A = torch.randn((500, 400), generator=gen, device=cuda, dtype=dt)
    A[3, 4] = float("nan")
    W, P = mak.left_polar(cm(A), precision="mixed")
    assert not ordinary(W).all() and not ordinary(P).all()
