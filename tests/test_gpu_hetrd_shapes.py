"""The Householder kernel (csrc/hetrd_reg.cu) at the edges of its launch shapes.

Every n at which the shape changes (rows per lane, warps per pair, columns in registers) and its
neighbours, against zhegv under the gates of test_gpu_parity.check; and matrices whose reflectors
are the identity (block-diagonal, diagonal), where v, w and tau are zero for whole steps.
"""
from __future__ import annotations

import numpy as np
import pytest

from oracle import metrics as Mx
from test_gpu_parity import check, run

pytestmark = pytest.mark.gpu

EDGES = sorted({m for e in (1, 8, 16, 24, 32, 40, 56, 64, 76, 84, 96, 128, 144) for m in (e, e + 1)} | {2, 3, 31, 55, 160})


def pair(rng, n, blocks=1):
    G = rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))
    H = rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))
    A, B = G + G.conj().T, np.eye(n) + H @ H.conj().T / n
    if blocks > 1:
        keep = (np.arange(n)[:, None] * blocks // n) == (np.arange(n)[None, :] * blocks // n)
        A, B = A * keep, np.eye(n)
    return A, B


@pytest.mark.parametrize("n", EDGES)
def test_every_shape(oracle_mod, n):
    rng = np.random.default_rng(n)
    ps = [pair(rng, n) for _ in range(4)] + [pair(rng, n, blocks=min(n, 3))]
    A = Mx.from_mats(np.array([p[0] for p in ps]))
    B = Mx.from_mats(np.array([p[1] for p in ps]).astype(np.complex128))
    W, X, info = run(n, A, B)
    Wr, Xr, ir = oracle_mod.hegv(A, B, n, nthreads=4)
    assert (ir == 0).all()
    check(A, B, W, X, info, Wr, Xr, n)
