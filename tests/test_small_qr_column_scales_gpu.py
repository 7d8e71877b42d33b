"""The one-CTA QR of blocks whose columns differ by many decades, in both
directions: the products of a reflector's column with the columns to its right
must neither overflow nor lose digits among the subnormals, whichever of the
two columns is the large one.

Householder QR is backward stable column by column: ||(A - QR) e_c|| <= a
modest multiple of n eps ||A e_c||; the residual is formed from the columns
scaled to 1 by powers of two.
"""

from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from conftest import to_dev, to_host

pytestmark = pytest.mark.gpu
# exponents of two of the even and the odd columns
SCALES = {8: [(98, 950), (-98, -960), (98, -1000), (-98, 990), (0, 700), (-990, 990)],
          4: [(18, 108), (-18, -120), (18, -120), (-18, 110), (0, 70), (-100, 100)]}
DTYPES = [np.float64, np.complex128, np.float32, np.complex64]


@pytest.mark.parametrize("dt", DTYPES, ids=lambda d: np.dtype(d).name)
@pytest.mark.parametrize("which", range(6))
@pytest.mark.parametrize("shape", [(64, 32), (128, 64), (37, 20), (5, 9), (8, 8), (150, 30)],
                         ids=lambda s: f"{s[0]}x{s[1]}")
@pytest.mark.parametrize("listed", [False, True])
def test_columns_of_mixed_scales(mak, cuda, dt, which, shape, listed):
    m, n = shape
    real = np.finfo(dt).dtype
    rng = np.random.default_rng(m + n)
    A = O.gaussian(rng, m, n, dt)
    e = np.array([SCALES[real.itemsize][which][c % 2] for c in range(n)])
    s = np.ldexp(np.ones(n), e)
    A = np.asfortranarray((A * s.astype(real)).astype(dt))
    call = mak.batched_qr_compact if listed else mak.batched_qr_compact_device
    (Q, R), = call([to_dev(A, cuda)])
    wide = np.complex128 if np.iscomplexobj(A) else np.float64
    Q, R = to_host(Q).astype(wide), to_host(R).astype(wide)
    assert np.isfinite(Q).all() and np.isfinite(R).all()
    A1, R1 = A.astype(wide) / s, R / s  # columns of ordinary size again
    bound = 8 * n * np.finfo(dt).eps
    assert np.all(np.linalg.norm(A1 - Q @ R1, axis=0) <= bound * np.linalg.norm(A1, axis=0))
    assert np.linalg.norm(Q.conj().T @ Q - np.eye(Q.shape[1])) <= bound
