"""The Newton-Schulz finish of the polar pullbacks' sign iteration (mixed
precision, from 384 columns): the batched call, which stops and switches on
the device, takes the steps of the single call, which looks from the host,
and both agree with the oracle, on both sides of the size where the finish
begins.  Bounds as for the batched pullbacks: 1e-10 against the oracle, 1e-13
between the two forms."""

from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from conftest import to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [np.float64, np.complex128], ids=["f64", "c128"])
def test_batched_finish_takes_the_single_calls_steps(mak, cuda, dt):
    rng = np.random.default_rng(305)
    blocks = [O.gaussian(rng, m, n, dt) for m, n in ((500, 383), (500, 384), (640, 417))]
    facs = [O.left_polar_svd(A) for A in blocks]
    cots = [(O.gaussian(rng, *W.shape, dt), O.gaussian(rng, *P.shape, dt)) for W, P in facs]
    dAs = [to_dev(np.zeros_like(A), cuda) for A in blocks]
    iters = []
    mak.batched_left_polar_pullback(dAs, [(to_dev(W, cuda), to_dev(P, cuda)) for W, P in facs],
                                    [(to_dev(a, cuda), to_dev(b, cuda)) for a, b in cots],
                                    precision="mixed", _info=iters)
    for i, (A, (W, P), (dW, dP), dA) in enumerate(zip(blocks, facs, cots, dAs)):
        ref = O.left_polar_pullback(np.zeros_like(A), A, W, P, dW, dP)
        assert O.rel_err(to_host(dA), ref) <= 1e-10, i
        d1 = to_dev(np.zeros_like(A), cuda)
        info = {}
        mak.left_polar_pullback_(d1, None, (to_dev(W, cuda), to_dev(P, cuda)),
                                 (to_dev(dW, cuda), to_dev(dP, cuda)), precision="mixed",
                                 _info=info)
        assert iters[i] == info["iterations"], i
        assert O.rel_err(to_host(dA), to_host(d1)) <= 1e-13, i
