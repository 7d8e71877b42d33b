"""The one-CTA QR's form for tall, narrow blocks and the rule that chooses it:
rows per column on both sides of the rule (alone on an SM: 6, in 32 bits 4;
many blocks: 16, and 128 to 512 rows), one column, one row more, blocks on both
sides of a third of an SM's shared memory, in lists of few and of many blocks
and of both forms.

Householder QR: ||A - QR|| / ||A|| and ||Q^H Q - I|| within a modest multiple
of eps times the column count.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DT = {"f64": torch.float64, "c64": torch.complex128, "f32": torch.float32, "c32": torch.complex64}
SHAPES = [(5, 1), (4, 1), (24, 4), (23, 4), (16, 4), (15, 4), (100, 2), (120, 20), (119, 20),
          (80, 20), (128, 8), (129, 8), (256, 16), (255, 16), (512, 4), (511, 4), (240, 50),
          (2000, 4), (3, 9), (40, 40), (1, 1)]


@pytest.mark.parametrize("dt", sorted(DT))
@pytest.mark.parametrize("copies", [1, 12])
@pytest.mark.parametrize("listed", [False, True])
def test_both_forms_in_one_list(mak, cuda, dt, copies, listed):
    gen = torch.Generator(device=cuda).manual_seed(copies)
    As = [torch.randn((n, m), generator=gen, device=cuda, dtype=DT[dt]).t()
          for _ in range(copies) for m, n in SHAPES]
    keep = [A.clone() for A in As]
    call = mak.batched_qr_compact if listed else mak.batched_qr_compact_device
    wide = torch.complex128 if As[0].is_complex() else torch.float64
    eps = torch.finfo(DT[dt]).eps
    for A, B, (Q, R) in zip(As, keep, call(As, positive=True)):
        assert torch.equal(A, B)
        m, n = A.shape
        k = min(m, n)
        Q, R, A = Q.to(wide), R.to(wide), A.to(wide)
        bound = 16 * max(n, 4) * eps
        assert float((Q @ R - A).norm()) <= bound * float(A.norm())
        assert float((Q.mH @ Q - torch.eye(k, device=cuda, dtype=wide)).norm()) <= bound
        assert bool((R.diagonal().real >= 0).all()) and torch.equal(R, R.triu())


def test_degenerate_tall_blocks(mak, cuda):
    A = torch.zeros((3, 200), device=cuda, dtype=torch.float64).t()
    (Q, R), = mak.batched_qr_compact_device([A])
    assert float(R.abs().max()) == 0.0
    assert float((Q.T @ Q - torch.eye(3, device=cuda, dtype=torch.float64)).norm()) <= 1e-14
    B = torch.from_numpy(np.asfortranarray(np.ones((400, 5)))).to(cuda).t().contiguous().t()
    B[:, 2] *= 1e200
    B[:, 3] *= 1e-200
    (Q, R), = mak.batched_qr_compact_device([B])
    assert bool(Q.isfinite().all()) and bool(R.isfinite().all())
    s = B[0]
    assert float(((Q @ (R / s) * s - B) / s).norm()) <= 1e-12
