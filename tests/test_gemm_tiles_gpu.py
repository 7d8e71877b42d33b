"""The native product at the edges of its tiles (16 x 16 and 32 x 32), of its
K step (32) and of its K splits, every op, against a 64-bit product.

Bound: an inner product of K terms summed in any order is within
(K + 2) eps sum |a||b| of the exact one (complex: four times that).
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

from conftest import to_dev, to_host

pytestmark = pytest.mark.gpu
# (1, 1, 1) .. one tile; 31/32/33 around a K step; tall K: split; many tiles: 32 x 32
SHAPES = [(1, 1, 1), (16, 16, 32), (17, 15, 33), (32, 33, 31), (31, 250, 1000), (5, 7, 4097),
          (700, 705, 40), (1500, 64, 96)]


@pytest.mark.parametrize("dt", [np.float64, np.complex128], ids=lambda d: np.dtype(d).name)
@pytest.mark.parametrize("ops", ["NN", "CN", "NC", "TT"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_native_gemm_tiles(mak, cuda, dt, ops, shape):
    from mak_gb300 import blas

    m, n, k = shape
    rng = np.random.default_rng(m + 7 * n + 13 * k)

    def rand(r, c):
        x = rng.standard_normal((r, c))
        return (x + 1j * rng.standard_normal((r, c)) if dt is np.complex128 else x).astype(dt)

    A = rand(m, k) if ops[0] == "N" else rand(k, m)
    B = rand(k, n) if ops[1] == "N" else rand(n, k)
    C0 = rand(m, n)
    f = {"N": lambda x: x, "T": lambda x: x.T, "C": lambda x: x.conj().T}
    a, b = f[ops[0]](A), f[ops[1]](B)
    C = to_dev(C0, cuda)
    blas.gemm(to_dev(A, cuda), to_dev(B, cuda), ops[0], ops[1], alpha=-1.0, beta=0.5, C=C)
    torch.cuda.synchronize()
    ref = -(a @ b) + 0.5 * C0
    eps = np.finfo(np.float64).eps
    bound = 4 * (k + 4) * eps * (np.abs(a) @ np.abs(b) + np.abs(C0))
    assert np.all(np.abs(to_host(C) - ref) <= 2 * bound)


@pytest.mark.parametrize("dt", [np.float32, np.complex64], ids=lambda d: np.dtype(d).name)
@pytest.mark.parametrize("shape", [(4100, 65), (3000, 320), (700, 690), (520, 515), (129, 96)],
                         ids=lambda s: f"{s[0]}x{s[1]}")
def test_fp32_tiles_through_qr(mak, cuda, dt, shape):
    """The FP32 tiles (32 x 128, 128 x 64, 64 x 64, 32 x 32 as the trailing
    matrix shrinks) with masks, splits and ragged edges, through a QR whose
    products they are; bound: backward stability, 170 eps sqrt(n)."""
    m, n = shape
    rng = np.random.default_rng(m)
    A = rng.standard_normal((m, n))
    A = (A + 1j * rng.standard_normal((m, n)) if dt is np.complex64 else A).astype(dt)
    for X in (A, np.asfortranarray(A.conj().T)):
        Q, R = mak.qr_compact(to_dev(X, cuda))
        Qh, Rh = to_host(Q).astype(np.complex128), to_host(R).astype(np.complex128)
        k = min(X.shape)
        bound = 2e-5 * np.sqrt(k)
        assert np.linalg.norm(X - Qh @ Rh) <= bound * np.linalg.norm(X)
        assert np.linalg.norm(Qh.conj().T @ Qh - np.eye(k)) <= bound * np.sqrt(k)


@pytest.mark.parametrize("dt", [np.float64, np.complex128], ids=lambda d: np.dtype(d).name)
@pytest.mark.parametrize("ops", ["NN", "CN", "NC", "TT"])
@pytest.mark.parametrize("k", [16, 127, 128, 129, 255, 256, 257, 511, 512, 513])
def test_split_operands_at_the_edges_of_one_pass(mak, cuda, dt, ops, k):
    """The split product where its operands' maxima and digits are formed in
    one pass (K up to 512, complex up to 256) and just beyond, ragged rows,
    rows of zeros and rows 2^200 apart; bound: 1e-13 of sum |a||b|, the split
    product's own."""
    from mak_gb300 import blas

    m, n = 77, 45
    rng = np.random.default_rng(k)

    def rand(r, c):
        x = rng.standard_normal((r, c))
        return (x + 1j * rng.standard_normal((r, c)) if dt is np.complex128 else x).astype(dt)

    a, b = rand(m, k), rand(k, n)
    a[5] = 0
    a[7] *= 2.0 ** 100
    a[8] *= 2.0 ** -100
    b[:, 3] = 0
    f = {"N": lambda x: x, "T": lambda x: x.T, "C": lambda x: x.conj().T}
    C = blas.gemm(to_dev(np.asfortranarray(f[ops[0]](a)), cuda),
                  to_dev(np.asfortranarray(f[ops[1]](b)), cuda), ops[0], ops[1],
                  precision="mixed")
    bound = 1e-13 * (np.abs(a) @ np.abs(b))
    assert np.all(np.abs(to_host(C) - a @ b) <= bound)
