"""Native products with more column tiles than one launch's grid has (65535 of
16 or 32 columns in Float64 and ComplexF64), through ``gemm`` and through the
QR of a matrix with millions of columns: the last columns before and the first
after a launch's end, and the ragged last tile.

The products of 40 terms are compared with the GPU's own 64-bit product in
sampled columns (40 eps of the operands' norms); the QR's columns by their
residual (a few eps per reflector).
"""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
EPS = torch.finfo(torch.float64).eps
EDGE = 32 * 65535


def cm(X):
    return X.t().contiguous().t()


def columns(n):
    at = torch.arange(0, n, 9973)
    edge = torch.arange(EDGE - 70, min(n, EDGE + 70))
    return torch.cat([at, edge[edge < n], torch.arange(n - 70, n)]).cuda()


@pytest.mark.parametrize("dt", [torch.float64, torch.complex128], ids=["f64", "c64"])
@pytest.mark.parametrize("m,n", [(17, EDGE + 33), (40, 2 * EDGE + 5)])
@pytest.mark.parametrize("op", ["N", "C"])
def test_gemm_columns(mak, cuda, dt, m, n, op):
    gen = torch.Generator(device=cuda).manual_seed(n)
    A = cm(torch.randn((m, 40), generator=gen, device=cuda, dtype=dt))
    B = torch.randn((n, 40), generator=gen, device=cuda, dtype=dt)
    C = cm(torch.randn((m, n), generator=gen, device=cuda, dtype=dt))
    cols = columns(n)
    ref = 2.0 * A @ (B[cols].mH if op == "C" else B[cols].mT) - 1.5 * C[:, cols]
    out = mak.gemm(A, cm(B) if op == "C" else B.t(), "N", op, alpha=2.0, beta=-1.5, C=C)
    err = (out[:, cols] - ref).norm(dim=0)
    assert bool((err <= 40 * EPS * (2 * A.norm() * B[cols].norm(dim=1) + 1.5 * ref.norm(dim=0))).all())


@pytest.mark.parametrize("dt,m,n", [(torch.float64, 33, 2_200_000), (torch.float64, 8, EDGE + 9),
                                    (torch.complex128, 17, EDGE + 100)])
def test_qr_of_millions_of_columns(mak, cuda, dt, m, n):
    gen = torch.Generator(device=cuda).manual_seed(m)
    A = torch.randn((n, m), generator=gen, device=cuda, dtype=dt).t()
    Q, R = mak.qr_compact(A)
    cols = columns(n)
    err = (Q @ R[:, cols] - A[:, cols]).norm(dim=0) / A[:, cols].norm(dim=0)
    assert float(err.max()) <= 8 * m * EPS
    assert float((Q.mH @ Q - torch.eye(m, device=cuda, dtype=dt)).norm()) <= 8 * m * EPS
