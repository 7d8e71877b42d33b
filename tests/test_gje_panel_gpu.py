"""The Gauss-Jordan panel at the edges of its launches, through left_polar of
square matrices (every Newton step inverts the iterate): one CTA and several,
ragged last CTAs and last panels, the largest cluster (4096 rows; ComplexF64
1536) and the first grid beyond it, rows that must be exchanged in every
column, and exact ties between pivot candidates.

||A - W P|| and ||W^H W - I|| are bounded by a modest multiple of n eps for
kappa up to 1e4 (Newton's iteration is backward stable); the bounds are
those of the polar tests, 1e-12 and 2e-5.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

from conftest import to_dev

pytestmark = pytest.mark.gpu
BOUND = {torch.float64: 1e-12, torch.complex128: 1e-12, torch.float32: 2e-5,
         torch.complex64: 2e-5}


def check(mak, A, bound, **kw):
    W, P = mak.left_polar(A, **kw)
    torch.cuda.synchronize()
    n = A.shape[0]
    assert float(torch.linalg.norm(A - W @ P) / torch.linalg.norm(A)) <= bound
    eye = torch.eye(n, dtype=A.dtype, device=A.device)
    assert float(torch.linalg.norm(W.mH @ W - eye)) <= bound * np.sqrt(n)


@pytest.mark.parametrize("dt", list(BOUND), ids=lambda d: str(d).split(".")[1])
@pytest.mark.parametrize("n", [1, 31, 33, 65, 300, 513, 1055])
def test_panel_sizes(mak, cuda, dt, n):
    gen = torch.Generator(device=cuda).manual_seed(n)
    A = torch.randn((n, n), generator=gen, device=cuda, dtype=dt).t()
    # a diagonal shift by a cyclic permutation: well conditioned, and the
    # largest entry of a column is never on the diagonal
    A = A / np.sqrt(n) + 4 * torch.roll(torch.eye(n, device=cuda, dtype=dt), 1, 0)
    check(mak, A.t().contiguous().t(), BOUND[dt])


@pytest.mark.parametrize("dt,n", [(torch.float64, 4096), (torch.float64, 4097),
                                  (torch.complex128, 1536), (torch.complex128, 1537)])
def test_largest_cluster_and_first_grid(mak, cuda, dt, n):
    gen = torch.Generator(device=cuda).manual_seed(n)
    A = torch.randn((n, n), generator=gen, device=cuda, dtype=dt)
    A = A / np.sqrt(n) + 4 * torch.roll(torch.eye(n, device=cuda, dtype=dt), 1, 0)
    check(mak, A.t().contiguous().t(), BOUND[dt], precision="mixed")


def test_tied_candidates(mak, cuda):
    """A Hadamard matrix: every candidate of the first column has the same
    magnitude, and its polar factor is itself over sqrt(n)."""
    H = np.array([[1.0]])
    while H.shape[0] < 256:
        H = np.block([[H, H], [H, -H]])
    A = to_dev(np.asfortranarray(H), cuda)
    W, P = mak.left_polar(A)
    assert float((W - A / 16).abs().max()) <= 1e-13
    assert float((P - 16 * torch.eye(256, device=cuda, dtype=A.dtype)).abs().max()) <= 1e-11


# Rows per CTA (16 CTAs) on both sides of the line from which a panel keeps
# multipliers that the row exchange's kernel finishes, ragged last panels, and
# the largest instance; matrices whose pivots move in every column.
@pytest.mark.parametrize("dt,n", [(torch.float64, 1792), (torch.float64, 1793), (torch.float64, 2049),
                                  (torch.complex128, 1280), (torch.complex128, 1281),
                                  (torch.complex128, 2500), (torch.float32, 2048),
                                  (torch.float32, 2055), (torch.complex64, 1664),
                                  (torch.complex64, 1665)])
def test_deferred_multipliers(mak, cuda, dt, n):
    gen = torch.Generator(device=cuda).manual_seed(n)
    Q, _ = mak.qr_compact(torch.randn((n, n), generator=gen, device=cuda, dtype=dt))
    Z, _ = mak.qr_compact(torch.randn((n, n), generator=gen, device=cuda, dtype=dt))
    d = torch.linspace(1, 100, n, device=cuda, dtype=torch.float64).to(dt)
    check(mak, Q @ (d[:, None] * Z.mH), BOUND[dt] * (1 if Q.real.dtype == torch.float64 else 5))


# The largest clusters of the other types and the first grid beyond them
# (ComplexF32 stops where 16 CTAs' rows no longer fit shared memory twice);
# W^H W = I and A = W P to n eps.
@pytest.mark.parametrize("dt,n", [(torch.float32, 4097), (torch.float32, 8192), (torch.float32, 8193),
                                  (torch.complex64, 4100), (torch.complex64, 7100),
                                  (torch.complex128, 2048), (torch.complex128, 2049)])
def test_largest_clusters_by_type(mak, cuda, dt, n):
    gen = torch.Generator(device=cuda).manual_seed(n)
    A = torch.randn((n, n), generator=gen, device=cuda, dtype=dt)
    A = A / np.sqrt(n) + 4 * torch.roll(torch.eye(n, device=cuda, dtype=dt), 1, 0)
    check(mak, A.t().contiguous().t(), n * torch.finfo(dt).eps, precision="mixed")
