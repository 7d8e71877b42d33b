"""The triangular inverse by doubling, through the QR pullback (dA = dQ R^-H
for dR = 0 after the projection) and the first Newton step of a tall polar:
one block, ragged last blocks and pairs without a partner, the levels below
and above the split products' width, and an exactly singular R.

The QR pullback at a well conditioned R (diagonal shifted) is within a modest
multiple of n eps cond(R) of the 64-bit formula: 1e-12 (Float64), 5e-4
(Float32) relative.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

import oracle as O
from conftest import to_dev, to_host

pytestmark = pytest.mark.gpu
TOL = {np.float64: 1e-12, np.complex128: 1e-12, np.float32: 5e-4, np.complex64: 5e-4}


@pytest.mark.parametrize("dt", list(TOL), ids=lambda d: np.dtype(d).name)
@pytest.mark.parametrize("n", [1, 31, 32, 33, 64, 97, 160, 300])
def test_qr_pullback_of_ragged_sizes(mak, cuda, dt, n):
    rng = np.random.default_rng(n)
    A = (O.gaussian(rng, n + 40, n, dt) / np.sqrt(n + 40) +
         2 * np.eye(n + 40, n)).astype(dt)
    Q, R = O.qr_compact(A)
    dQ, dR = O.gaussian(rng, n + 40, n, dt), O.gaussian(rng, n, n, dt)
    # real diagonal of the antihermitian part: gauge-invariant cotangents
    dA = to_dev(np.zeros_like(A), cuda)
    mak.qr_pullback_(dA, None, (to_dev(Q, cuda), to_dev(R, cuda)),
                     (to_dev(dQ, cuda), to_dev(dR, cuda)))
    w = np.complex128 if np.iscomplexobj(A) else np.float64
    Qw, Rw, dQw, dRw = (X.astype(w) for X in (Q, R, dQ, np.triu(dR)))
    M = Rw @ dRw.conj().T - dQw.conj().T @ Qw
    H = np.tril(M, -1)
    H = H + H.conj().T + np.diag(np.diag(M).real)
    ref = np.linalg.solve(Rw, (dQw + Qw @ H).conj().T).conj().T
    assert O.rel_err(to_host(dA), ref) <= TOL[dt]


@pytest.mark.parametrize("n", [257, 600, 1100])
def test_split_levels(mak, cuda, n):
    """Mixed precision: levels of 256 and wider as split products."""
    gen = torch.Generator(device=cuda).manual_seed(n)
    A = torch.randn((n, n + 64), generator=gen, device=cuda, dtype=torch.float64).t() / n ** 0.5
    A = A + 3 * torch.eye(n + 64, n, device=cuda, dtype=torch.float64)
    A = A.t().contiguous().t()
    d = [torch.randn((n, r), generator=gen, device=cuda, dtype=torch.float64).t()
         for r in (n + 64, n)]
    Q, R = mak.qr_compact(A)
    out = []
    for prec in ("native", "mixed"):
        dA = torch.zeros_like(A.t()).t()
        mak.qr_pullback_(dA, None, (Q, R), tuple(d), precision=prec)
        out.append(dA)
    assert float(torch.linalg.norm(out[0] - out[1]) / torch.linalg.norm(out[0])) <= 1e-12


def test_polar_of_a_rank_deficient_tall_matrix(mak, cuda):
    """R with a zero on its diagonal: the first iterate is exactly singular."""
    A = np.zeros((50, 20))
    A[:20] = np.triu(np.random.default_rng(0).standard_normal((20, 20)))
    A[7, 7:] = 0.0
    with pytest.raises(mak.polar.SingularException):
        mak.left_polar(to_dev(A, cuda))
