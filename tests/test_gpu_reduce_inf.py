"""An infinite diagonal entry of B, as zpotrf and ztrsm take it: that row of L is zero but for an infinite
pivot, the component drops out of the problem and leaves the eigenvalue 0.

Expected: the eigenvalues of the pair without that row and column, and a zero.  Bound: 64 n eps times the largest
(Cholesky, reduction and Householder of a well-conditioned pair).
"""
from __future__ import annotations

import numpy as np
import pytest

from oracle import metrics as Mx
from test_gpu_parity import run

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


# every number of 8-row blocks up to n = 56 and both kinds of block counts above, n > 144's other kernel
@pytest.mark.parametrize("n", [1, 3, 8, 16, 24, 32, 40, 47, 54, 64, 72, 80, 88, 96, 112, 128, 144, 160])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_infinite_pivot(n, precision):
    rng = np.random.default_rng(n)
    where = sorted({0, n // 2, n - 1})
    G = rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))
    A = G + G.conj().T
    B = np.eye(n) + 0.01 * A / np.sqrt(n)
    As, Bs, ref = [], [], []
    for k in where:
        keep = np.delete(np.arange(n), k)
        M = B.copy()
        M[k, k] = np.inf
        As.append(A)
        Bs.append(M)
        L = np.linalg.cholesky(B[np.ix_(keep, keep)])
        Li = np.linalg.inv(L) if n > 1 else L
        ref.append(np.sort(np.append(np.linalg.eigvalsh(Li @ A[np.ix_(keep, keep)] @ Li.conj().T) if n > 1 else [], 0.0)))
    W, X, info = run(n, Mx.from_mats(np.array(As)), Mx.from_mats(np.array(Bs)), precision)
    assert (info == 0).all() and np.isfinite(X).all()
    for w, r, x, k in zip(W, ref, X, where):
        assert np.abs(w - r).max() <= 64 * n * EPS * max(np.abs(r).max(), np.abs(A).max() if n == 1 else 0.0)
        assert (x.reshape(n, n).T[k] == 0).all()
