"""The eigenvalue search of csrc/tridiag.cu runs until every bracket is closed.

T = tridiag(1, h |i - c|, 1) is two mirrored, weakly coupled ramps: its eigenvalues come in pairs that
agree to anything between a few digits and all of them, so that det(T - x I) is close to zero at an end
of many brackets and every chord lands on that end.  A search that stopped after 128 counts returned
eigenvalues of these T 30 to 182 u ||T|| off, with info = 0 (their vectors pass the residual test).

A = T (real tridiagonal, exact in FP64) and B = I leave T as it is: every reflector is the identity.
What is left is the search itself, bounded independently of n by 8 u ||T||, u = 2^-53: the counts are
those of a T whose entries are off by at most 2 u ||T|| (d - x), 2 u ||T|| (the rounding of the fused
multiply-add) on the diagonal and 1.5 u |e| (e^2, its product, the sum) twice a row off it, and half of
the last bracket is at most u ||T||.  The reference is bisection in 80-bit arithmetic.
"""
from __future__ import annotations

import numpy as np
import pytest

from oracle import metrics as Mx
from test_gpu_parity import run

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def eigenvalues(d):
    """Eigenvalues of tridiag(1, d[p], 1) for every p, by bisection in extended precision."""
    d = np.asarray(d, np.longdouble)
    b, n = d.shape
    j = np.arange(n)[None, :]
    hi = np.broadcast_to(np.abs(d).max(axis=1)[:, None] + 2.5, (b, n)).copy()
    lo = -hi
    for _ in range(76):
        x = (lo + hi) / 2
        q = d[:, :1] - x
        below = (q < 0).astype(np.int64)
        for i in range(1, n):
            q = d[:, i:i + 1] - x - 1 / np.where(q == 0, np.longdouble(1e-40), q)
            below += q < 0
        hi = np.where(below > j, x, hi)
        lo = np.where(below > j, lo, x)
    return (lo + hi) / 2


@pytest.mark.parametrize("n,h,c", [(56, 1.0, 29.5), (57, 1.0, 29.5), (59, 1.0, 29.5), (60, 0.75, 33.5),
                                   (63, 0.75, 35.5), (67, 1.0, 39.0), (68, 1.0, 39.5), (77, 0.25, 39.0)])
def test_bracket_beside_another_eigenvalue(n, h, c):
    d = (h * np.abs(np.arange(n) - c))[None]
    T = np.diag(d[0]) + np.diag(np.ones(n - 1), 1) + np.diag(np.ones(n - 1), -1)
    W, _, info = run(n, Mx.from_mats(T[None].astype(np.complex128)), Mx.from_mats(np.eye(n, dtype=np.complex128)[None]))
    ref = eigenvalues(d)
    assert info[0] == 0 and (np.diff(W[0]) >= 0).all()
    assert np.abs(W - ref).max() <= 8 * U * np.abs(ref).max(), float(np.abs(W - ref).max() / np.abs(ref).max() / U)
