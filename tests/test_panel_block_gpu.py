"""The QR panel's block round (all columns of a panel from one Gram matrix)
and the column-by-column path it leaves the panel to, at the edges of its
rule: the fewest rows and columns that try it, ragged panels, the cluster and
grid launches, and panels whose columns are (nearly) dependent or out of the
squared norms' range.

Householder QR is backward stable: ||A - QR|| / ||A|| and ||Q^H Q - I|| are
bounded by a modest multiple of eps whatever the conditioning, so the bounds
below (450 eps in Float64, 170 eps in Float32, with the square root of the
column count) hold on both paths.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

import oracle as O
from conftest import to_dev, to_host

pytestmark = pytest.mark.gpu
DTYPES = [np.float64, np.complex128, np.float32, np.complex64]
TOL = {np.float64: 1e-13, np.complex128: 1e-13, np.float32: 2e-5, np.complex64: 2e-5}
# rows x columns: 3 rows per column is the fewest that tries the block round,
# 8 columns the narrowest panel; 2048 rows the last cluster launch
SHAPES = [(24, 8), (21, 7), (96, 32), (95, 32), (97, 33), (130, 41), (513, 31), (2048, 64),
          (2049, 40), (5000, 63)]


def make(kind, m, n, dt):
    rng = np.random.default_rng(1000 * m + n)
    A = O.gaussian(rng, m, n, dt)
    eps = np.finfo(dt).eps
    if kind == "dependent":  # two columns equal up to a few eps: the norm test refuses
        A[:, n // 2] = A[:, 1] * dt(2) + A[:, n // 2] * dt(4 * eps)
    elif kind == "ramp":  # every column mostly along the first one
        A = (A * dt(0.01) + A[:, :1]).astype(dt)
    elif kind == "scaled":  # squared norms over and under the range
        s = 1e170 if np.dtype(dt).itemsize // (2 if np.iscomplexobj(A) else 1) == 8 else 1e16
        A[:, 2] *= dt(s)
        A[:, n - 1] *= dt(1 / s)
    elif kind == "triangular":  # zero below the diagonal: beta_j = -alpha_j
        A = np.triu(A).astype(dt)
    return np.asfortranarray(A)


@pytest.mark.parametrize("dt", DTYPES, ids=lambda d: np.dtype(d).name)
@pytest.mark.parametrize("kind", ["gaussian", "dependent", "ramp", "scaled", "triangular"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: f"{s[0]}x{s[1]}")
def test_block_round_and_fallback(mak, cuda, dt, kind, shape):
    m, n = shape
    A = make(kind, m, n, dt)
    Q, R = mak.qr_compact(to_dev(A, cuda))
    torch.cuda.synchronize()
    Qh, Rh = to_host(Q), to_host(R)
    wide = np.complex128 if np.iscomplexobj(A) else np.float64
    Aw, Qw, Rw = A.astype(wide), Qh.astype(wide), Rh.astype(wide)
    bound = TOL[dt] * np.sqrt(n)
    # column-wise residual: the columns' scales may differ by many decades
    scale = np.abs(Aw).max(axis=0)
    err = np.linalg.norm((Aw - Qw @ Rw) / scale, axis=0)
    assert np.all(err <= bound * np.linalg.norm(Aw / scale, axis=0))
    assert np.linalg.norm(Qw.conj().T @ Qw - np.eye(n)) <= bound * np.sqrt(n)
    d = np.diagonal(Rh)
    assert np.all(d.real >= 0) and np.all(d.imag == 0)
    assert np.array_equal(np.triu(Rh), Rh)
    if kind == "gaussian":
        Ro = O.qr_compact(A)[1]
        assert O.rel_err(Rh, Ro) <= (1e-12 if TOL[dt] < 1e-10 else 2e-5)


# The tallest 32-column panels of a 152-SM GPU: rows per CTA that fill the
# shared memory beside the panel kernel's static arrays.  There the block
# round's own scratch does not fit and the column rounds take over.
TALLEST = {"f64": 152 * 838, "c64": 152 * 388, "f32": 152 * 1742, "c32": 152 * 840}


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", sorted(TALLEST))
def test_tallest_panels_are_accepted(mak, dtype):
    if torch.cuda.get_device_properties(0).multi_processor_count < 152:
        pytest.skip("needs 152 SMs")
    td = {"f64": torch.float64, "c64": torch.complex128, "f32": torch.float32,
          "c32": torch.complex64}[dtype]
    gen = torch.Generator(device="cuda").manual_seed(5)
    A = torch.randn(TALLEST[dtype], 32, dtype=td, device="cuda", generator=gen)
    Q, R = mak.qr_compact(A)
    eps = torch.finfo(td).eps
    # backward error of 32 reflectors: a few eps times the column count
    assert (Q @ R - A).norm() <= 32 * 8 * eps * A.norm()
    assert (Q.mH @ Q - torch.eye(32, dtype=td, device="cuda")).norm() <= 32 * 8 * eps
