"""Wide native products of few rows and a short K, at the edges of their tiles:
rows 1 .. 33 around 16 and 32, K around 8, 16 and 32 (a step of K that is not
padded any more), and the T-factor product of panels of 1 .. 33 rows (8, 16 or
32 rows of threads) through the QR of wide matrices.

A product of K terms is within K eps of |A| |B|; the QR's columns within a few
eps per reflector.
"""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DT = {"f64": torch.float64, "c64": torch.complex128, "f32": torch.float32, "c32": torch.complex64}


def cm(X):
    return X.t().contiguous().t()


@pytest.mark.parametrize("dt", ["f64", "c64"])
@pytest.mark.parametrize("M", [1, 8, 16, 17, 33])
@pytest.mark.parametrize("K", [1, 3, 8, 9, 31, 33, 65])
@pytest.mark.parametrize("op", ["N", "C"])
def test_wide_products(mak, cuda, dt, M, K, op):
    gen = torch.Generator(device=cuda).manual_seed(100 * M + K)
    N = 20011
    A = torch.randn((M, K), generator=gen, device=cuda, dtype=DT[dt])
    B = torch.randn((K, N), generator=gen, device=cuda, dtype=DT[dt])
    C = torch.randn((M, N), generator=gen, device=cuda, dtype=DT[dt])
    o = (lambda X: cm(X.mH.resolve_conj())) if op == "C" else cm
    out = mak.gemm(o(A), o(B), op, op, alpha=-1.0, beta=1.0, C=cm(C.clone()))
    bound = 4 * (K + 1) * torch.finfo(DT[dt]).eps * (A.abs() @ B.abs() + C.abs())
    assert bool(((out - (C - A @ B)).abs() <= bound).all())


@pytest.mark.parametrize("dt", sorted(DT))
@pytest.mark.parametrize("m", [1, 3, 8, 9, 16, 17, 32, 33, 40])
def test_qr_of_few_rows(mak, cuda, dt, m):
    gen = torch.Generator(device=cuda).manual_seed(m)
    A = torch.randn((60001, m), generator=gen, device=cuda, dtype=DT[dt]).t()
    Q, R = mak.qr_compact(A)
    wide = torch.complex128 if A.is_complex() else torch.float64
    eps = torch.finfo(DT[dt]).eps
    Q, R, A = Q.to(wide), R.to(wide), A.to(wide)
    err = (Q @ R - A).norm(dim=0) / A.norm(dim=0)
    assert float(err.max()) <= 16 * max(m, 4) * eps
    assert float((Q.mH @ Q - torch.eye(m, device=cuda, dtype=wide)).norm()) <= 16 * max(m, 4) * eps
    assert torch.equal(R, R.triu())
