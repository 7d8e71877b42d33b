"""Mixed-precision QR whose 128-wide block reflectors are merged (m n >= 4e6):
ragged last blocks of every kind (less than a panel, one block, more than one,
more than two), wide and tall, full and compact, with the look-ahead.

The split products are good to 1e-13 of sum |a||b| (their test's bound), and
a factorization applies about n / 256 of them to every entry, so 5e-13
relative bounds R (against the oracle), the residual and the columns of
Q^H Q - I, as for the 128-wide blocking.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

import oracle as O
from conftest import to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,dt,full", [
    (8000, 520, np.float64, False), (4100, 1000, np.float64, False),
    (2100, 1930, np.float64, False), (2000, 2100, np.float64, False),
    (2050, 1960, np.float64, True), (6500, 640, np.complex128, False),
    (3000, 1345, np.complex128, False)],
    ids=lambda v: str(v) if not isinstance(v, type) else np.dtype(v).name)
def test_merged_block_reflectors(mak, cuda, m, n, dt, full):
    rng = np.random.default_rng(m + n)
    A = O.gaussian(rng, m, n, dt)
    Ad = to_dev(A, cuda)
    Q, R = (mak.qr_full if full else mak.qr_compact)(Ad, precision="mixed")
    torch.cuda.synchronize()
    k = min(m, n)
    Ro = O.qr_compact(A)[1]
    Rh = to_host(R)
    assert O.rel_err(Rh[:k], Ro) <= 5e-13
    assert np.array_equal(np.triu(Rh), Rh)
    assert float(torch.linalg.norm(Q @ R - Ad) / torch.linalg.norm(Ad)) <= 5e-13
    eye = torch.eye(Q.shape[1], dtype=Q.dtype, device=cuda)
    assert float(torch.linalg.norm(Q.mH @ Q - eye)) <= 5e-13 * np.sqrt(Q.shape[1])


@pytest.mark.parametrize("dt", [np.float64, np.complex128], ids=lambda d: np.dtype(d).name)
@pytest.mark.parametrize("blocksize", [0, 5, 24, 31])
def test_t_factor_from_panels(mak, cuda, dt, blocksize):
    """The 128-wide T factor from panels whose width does not divide 128."""
    rng = np.random.default_rng(blocksize)
    A = O.gaussian(rng, 700, 300, dt)
    Ad = to_dev(A, cuda)
    Q, R = mak.qr_compact(Ad, precision="mixed", blocksize=blocksize)
    assert O.rel_err(to_host(R), O.qr_compact(A)[1]) <= 5e-13
    assert O.qr_residual(A, to_host(Q), to_host(R)) <= 5e-13
    assert O.orth_error(to_host(Q)) <= 5e-13 * np.sqrt(300)
