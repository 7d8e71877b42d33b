"""Panels on which the block round must not be taken: every column keeps more
than half its squared norm after the columns before it are projected out, yet
the dependence builds up over the panel (condition numbers of 25 to 10^4).

The round is taken only if the inverse of the panel's factor, columns scaled
to norm one, has a squared Frobenius norm of at most 2 per column, so an
accepted 32-column panel loses at most 64 eps of orthogonality to its Gram
matrix; Householder reflectors themselves lose a few eps per sqrt(column).
The bound below is 100 eps in the 2-norm per panel of 32 columns.
"""

from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from conftest import to_dev, to_host

pytestmark = pytest.mark.gpu
DTYPES = [np.float64, np.complex128, np.float32, np.complex64]
# (kept share of the squared norm, rows above the diagonal that hold the rest;
# 0: all of them)
KINDS = [(0.8, 0), (0.7, 0), (0.6, 0), (0.51, 0), (0.51, 1), (0.6, 2), (0.55, 3), (0.7, 4),
         (0.55, 4)]


def dependent(rng, m, n, keep, band, dt):
    """U R with orthonormal U; R_jj^2 = keep, the rest spread with one sign over
    the rows above (the inverse then adds up instead of cancelling)."""
    R = np.eye(n)
    for j in range(1, n):
        k = min(j, band) if band else j
        R[j, j] = np.sqrt(keep)
        R[j - k:j, j] = -np.sqrt((1 - keep) / k)
    wide = np.complex128 if np.dtype(dt).kind == "c" else np.float64
    U = np.linalg.qr(O.gaussian(rng, m, n, wide))[0]
    return U @ R


def check(A, Q, R, n):
    eps = np.finfo(A.dtype).eps
    wide = np.complex128 if A.dtype.kind == "c" else np.float64
    Aw, Qw, Rw = A.astype(wide), Q.astype(wide), R.astype(wide)
    bound = 100 * eps * np.ceil(n / 32)
    assert np.linalg.norm(Qw.conj().T @ Qw - np.eye(Q.shape[1]), 2) <= bound
    assert np.linalg.norm(Aw - Qw @ Rw, 2) <= bound * np.linalg.norm(Aw, 2)


@pytest.mark.parametrize("dt", DTYPES, ids=lambda d: np.dtype(d).name)
@pytest.mark.parametrize("kind", KINDS, ids=lambda k: f"{k[0]}-{k[1]}")
@pytest.mark.parametrize("shape", [(96, 32), (400, 32), (401, 33), (60, 20), (2500, 64)],
                         ids=lambda s: f"{s[0]}x{s[1]}")
def test_dependence_over_a_panel(mak, cuda, dt, kind, shape):
    rng = np.random.default_rng(11)
    A = np.asfortranarray(dependent(rng, *shape, *kind, dt).astype(dt))
    Q, R = mak.qr_compact(to_dev(A, cuda))
    check(A, to_host(Q), to_host(R), shape[1])


@pytest.mark.parametrize("dt", [np.float64, np.complex128], ids=lambda d: np.dtype(d).name)
@pytest.mark.parametrize("at", [0, 64, 150])
def test_dependent_columns_inside_a_wider_matrix(mak, cuda, dt, at):
    rng = np.random.default_rng(12)
    A = O.gaussian(rng, 1100, 300, dt) / np.sqrt(1100)
    A[:, at:at + 32] = dependent(rng, 1100, 32, 0.55, 4, dt)
    A = np.asfortranarray(A)
    Q, R = mak.qr_compact(to_dev(A, cuda), precision="mixed")
    check(A, to_host(Q), to_host(R), 300)
    L, Q = mak.lq_compact(to_dev(np.asfortranarray(A.conj().T), cuda))
    check(A, to_host(Q).conj().T, to_host(L).conj().T, 300)


@pytest.mark.parametrize("dt", [np.float64, np.complex64], ids=lambda d: np.dtype(d).name)
def test_isometries_that_inherit_the_panels(mak, cuda, dt):
    rng = np.random.default_rng(13)
    A = np.asfortranarray(dependent(rng, 500, 32, 0.6, 2, dt).astype(dt))
    wide = np.complex128 if np.dtype(dt).kind == "c" else np.float64
    eps = np.finfo(dt).eps
    W = to_host(mak.left_polar(to_dev(A, cuda))[0]).astype(wide)
    N = to_host(mak.qr_null(to_dev(A, cuda))).astype(wide)
    Q = to_host(mak.batched_qr_compact([to_dev(A, cuda)] * 2)[1][0]).astype(wide)
    # W = Q X: the polar iteration's own tolerance, eps^(2/3), squared by its last step
    for X in (W, N, Q):
        assert np.linalg.norm(X.conj().T @ X - np.eye(X.shape[1]), 2) <= 200 * eps
    assert np.linalg.norm(N.conj().T @ A) <= 200 * eps * np.linalg.norm(A)
