"""The device work lists read their inputs in place where they may: the
records' layout, the overlap test that falls back to copies (CPU), and inputs
in every layout, lazily conjugated, or sharing memory with the outputs (GPU)."""

from __future__ import annotations

import ctypes as ct

import numpy as np
import pytest
import torch

import oracle as O
from conftest import to_host


def cm(m, n, dtype=torch.float64, ld=None, device="cpu"):
    return torch.randn((n, ld or m), dtype=dtype, device=device).t()[:m]


def test_records_match_the_c_struct(mak):
    from mak_gb300 import _lib, batched

    As = [cm(5, 3), cm(7, 2, torch.complex128, ld=9), cm(4, 6, torch.float32), cm(1, 1)]
    outs = [(cm(A.shape[0], min(A.shape), A.dtype), cm(min(A.shape), A.shape[1], A.dtype))
            for A in As]
    outs[2] = (outs[2][0], None)
    rec = batched._item_records(As, outs)
    assert rec.nbytes == len(As) * ct.sizeof(_lib.mak_batch_item)
    for it, A, (Q, R) in zip(batched._items(As, outs), As, outs):
        assert (it.m, it.n) == tuple(A.shape) and it.A == A.data_ptr() and it.Q == Q.data_ptr()
        assert it.R == (R.data_ptr() if R is not None else None)
        assert it.dtype == batched.DTYPE_CODE[A.dtype] and it.reserved == 0
        assert it.lda == (9 if it.m == 7 else it.m) and it.ldq == Q.shape[0]


@pytest.mark.parametrize("m,n", [(6, 4), (4, 6), (1, 5), (5, 1)])
def test_overlap_rule(mak, m, n):
    from mak_gb300 import batched

    k = min(m, n)
    buf = torch.zeros(400, dtype=torch.float64)

    def at(off, r, c):
        return buf[off:off + r * c].view(c, r).t()

    far = (at(200, m, k), at(300, k, n))
    # input right before / after the outputs, then one element into them
    for off, hit in ((200 - m * n, False), (200 - m * n + 1, True), (200 + m * k, False),
                     (200 + m * k - 1, True), (300 + k * n, False), (300 + k * n - 1, True)):
        rec = batched._item_records([at(off, m, n), at(0, 1, 1)], [far, (at(398, 1, 1), None)])
        assert batched._overlaps(rec, True) is hit, off


@pytest.mark.gpu
@pytest.mark.parametrize("dt", [torch.float64, torch.complex64], ids=["d", "c"])
def test_inputs_in_any_layout(mak, cuda, dt):
    base = [cm(40, 12, dt, device=cuda), cm(30, 20, dt, ld=50, device=cuda),
            torch.randn((25, 10), dtype=dt, device=cuda),          # row-major
            cm(9, 33, dt, device=cuda).mH,                         # conjugate transpose
            torch.randn((60, 40), dtype=dt, device=cuda)[::2, ::3],
            torch.randn((1, 7), dtype=dt, device=cuda), torch.randn((7, 1), dtype=dt, device=cuda)]
    keep = [to_host(A.resolve_conj()).copy() for A in base]
    tol = 1e-12 if dt == torch.float64 else 2e-5
    outs = mak.batched_qr_compact_device(base)
    tall = [A for A in base if A.shape[0] >= A.shape[1]]
    polars = mak.batched_left_polar_device(tall)
    for A, H, (Q, R) in zip(base, keep, outs):
        assert np.array_equal(to_host(A.resolve_conj()), H)
        assert O.rel_err(to_host(R), O.qr_compact(H)[1]) <= tol
        assert O.qr_residual(H, to_host(Q), to_host(R)) <= tol
    for A, (W, P) in zip(tall, polars):
        assert float(torch.linalg.norm(A - W @ P)) <= tol * float(torch.linalg.norm(A)) * 10


@pytest.mark.gpu
def test_outputs_over_the_inputs(mak, cuda):
    """With copy_inputs (the default) outputs may reuse the inputs' memory."""
    A, B = cm(24, 10, device=cuda), cm(30, 10, device=cuda)
    H = [to_host(A).copy(), to_host(B).copy()]
    R = [cm(10, 10, device=cuda), cm(10, 10, device=cuda)]
    # A's factor goes over B and the other way round
    Q = [B[:24], torch.as_strided(A, (10, 10), (1, 24))]
    outs = mak.batched_qr_compact_device([A, B[:, :10][:10]], outs=[(Q[0], R[0]), (Q[1], R[1])])
    for h, (q, r) in zip((H[0], H[1][:10]), outs):
        assert O.qr_residual(h, to_host(q), to_host(r)) <= 1e-13
