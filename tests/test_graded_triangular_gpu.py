"""The triangular inverse of graded factors (columns or rows of R scaled over
many decades) and of the factors of smooth columns, through the QR pullback and
the first Newton step of a tall polar: below and above the size from which the
pivoted elimination takes over in mixed precision.

|X| |R| |X| of an inverse X bounds its error componentwise in n eps, and
neither scaling changes its ratio to |X|; so the pullback dA = dQ R^-H has to
reach, column by column, what that bound gives for the unscaled factor.
"""

from __future__ import annotations

import numpy as np
import pytest
import scipy.linalg as sl
import torch

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


def gauss(gen, m, n, dt):
    return torch.randn((m, n), generator=gen, device="cuda", dtype=dt)


def cm(X):
    return X.t().contiguous().t()


def graded(kind, n, dt):
    gen = torch.Generator(device="cuda").manual_seed(n)
    R = torch.triu(torch.linalg.qr(gauss(gen, 2 * n, n, dt))[1])
    s = 10.0 ** (16 * (torch.rand(n, generator=gen, device="cuda", dtype=torch.float64) - 0.5))
    if kind == "columns":
        return gen, R, R * s
    return gen, R, R * torch.logspace(0, -10, n, device="cuda", dtype=torch.float64)[:, None]


@pytest.mark.parametrize("kind", ["columns", "rows"])
@pytest.mark.parametrize("dt,n", [(torch.float64, 257), (torch.float64, 700),
                                  (torch.complex128, 300), (torch.complex128, 520)])
def test_qr_pullback_of_graded_factors(mak, cuda, kind, dt, n):
    gen, R0, R = graded(kind, n, dt)
    m = n + 60
    Q = torch.linalg.qr(gauss(gen, m, n, dt))[0]
    dQ = gauss(gen, m, n, dt)
    for _ in range(2):  # orthogonal to Q: dA = dQ R^-H
        dQ = dQ - Q @ (Q.mH @ dQ)
    dA = cm(torch.zeros((m, n), device="cuda", dtype=dt))
    mak.qr_pullback_(dA, None, (cm(Q), cm(R)), (cm(dQ), None), rank_atol=0.0, precision="mixed")
    ref = sl.solve_triangular(R.cpu().numpy(), dQ.mH.resolve_conj().cpu().numpy()).conj().T
    err = np.linalg.norm(dA.cpu().numpy() - ref, axis=0) / np.linalg.norm(ref, axis=0)
    R0 = R0.cpu().numpy()
    X0 = np.abs(sl.solve_triangular(R0, np.eye(n)))
    amp = np.max(np.linalg.norm(X0 @ np.abs(R0) @ X0, axis=1) / np.linalg.norm(X0, axis=1))
    assert err.max() <= n * EPS * amp


@pytest.mark.parametrize("precision", ["native", "mixed"])
@pytest.mark.parametrize("dt,n", [(torch.float64, 60), (torch.float64, 100),
                                  (torch.complex128, 90), (torch.float64, 300)])
def test_qr_pullback_of_smooth_columns(mak, cuda, precision, dt, n):
    """Trailing blocks of R far smaller than what stands above them: inverses
    multiplied block by block would cancel (condition 10^5 to 10^10)."""
    gen = torch.Generator(device="cuda").manual_seed(n)
    t = torch.linspace(-1, 1, 2 * n, device="cuda", dtype=torch.float64)
    s = torch.linspace(-1, 1, n, device="cuda", dtype=torch.float64)
    K = torch.exp(-(((t[:, None] - s[None, :]) * n / 6) ** 2)).to(dt)
    R = torch.triu(torch.linalg.qr(K)[1])
    m = n + 60
    Q = torch.linalg.qr(gauss(gen, m, n, dt))[0]
    dQ = gauss(gen, m, n, dt)
    for _ in range(2):
        dQ = dQ - Q @ (Q.mH @ dQ)
    dA = cm(torch.zeros((m, n), device="cuda", dtype=dt))
    mak.qr_pullback_(dA, None, (cm(Q), cm(R)), (cm(dQ), None), rank_atol=0.0,
                     precision=precision)
    Rh, dh = R.cpu().numpy(), dQ.cpu().numpy()
    X = np.abs(sl.solve_triangular(Rh, np.eye(n)))
    ref = sl.solve_triangular(Rh, dh.conj().T).conj().T
    # both sides carry the substitution's error: rows of |X| |R| |X| times |dQ|
    bound = 2 * n * EPS * np.linalg.norm(X @ np.abs(Rh) @ X @ np.abs(dh).T)
    assert np.linalg.norm(dA.cpu().numpy() - ref) <= bound


@pytest.mark.parametrize("kind", ["columns", "rows"])
@pytest.mark.parametrize("dt,n", [(torch.float64, 600), (torch.complex128, 300)])
def test_tall_polar_of_graded_factors(mak, cuda, kind, dt, n):
    gen, _, R = graded(kind, n, dt)
    Q = torch.linalg.qr(gauss(gen, n + 100, n, dt))[0]
    A = cm(Q @ R)
    W, P = mak.left_polar(A, precision="mixed", maxiter=60)
    eye = torch.eye(n, device="cuda", dtype=dt)
    # the iteration's tolerance eps^(2/3) squared by its last step, sqrt(n) of them
    assert float((W.mH @ W - eye).norm()) <= 1e-11
    assert float((A - W @ P).norm() / A.norm()) <= 1e-12


@pytest.mark.parametrize("n", [3584, 3585])
def test_both_sides_of_the_elimination(mak, cuda, n):
    gen = torch.Generator(device="cuda").manual_seed(n)
    R = torch.triu(gauss(gen, n, n, torch.float64)) / n ** 0.5
    R = cm(R + 2 * torch.eye(n, device="cuda", dtype=torch.float64))
    Q = cm(torch.eye(n + 8, n, device="cuda", dtype=torch.float64))
    dQ = torch.zeros((n, n + 8), device="cuda", dtype=torch.float64).t()
    dQ[n:] = gauss(gen, 8, n, torch.float64)
    dA = torch.zeros((n, n + 8), device="cuda", dtype=torch.float64).t()
    mak.qr_pullback_(dA, None, (Q, R), (dQ, None), rank_atol=0.0, precision="mixed")
    # cond(R) is a modest number; rows of the products of n terms: n eps
    assert float((dA @ R.mT - dQ).norm()) <= n * EPS * float(dA.norm() * R.norm())
