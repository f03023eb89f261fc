"""The tensor-core Cholesky and reduction (csrc/reduce_dmma.cu) at the edges of its blocks.

A leading minor that is not positive definite must be reported at zpotrf's order wherever it falls in
the 8-row blocks (first and last row of a block, the padded last block, rows held by the second warp of
a column block), and the pairs beside it must be solved; a NaN in B is reported as LAPACK's zpotrf does
(the first minor it makes non-positive).
"""
from __future__ import annotations

import numpy as np
import pytest

from oracle import metrics as Mx
from test_gpu_hetrd_shapes import pair
from test_gpu_parity import check, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 7, 8, 9, 40, 54, 56, 57, 72, 84, 96, 105, 128, 144, 150])
def test_info_of_the_first_bad_minor(oracle_mod, n):
    rng = np.random.default_rng(n)
    at = sorted({0, min(7, n - 1), min(8, n - 1), min(33, n - 1), n // 2, n - 1})
    ps = [pair(rng, n) for _ in range(len(at) + 2)]
    A = Mx.from_mats(np.array([p[0] for p in ps]))
    Bm = np.array([p[1] for p in ps]).astype(np.complex128)
    for p, k in enumerate(at):
        Bm[p, k, k] = -1.0
    Bm[len(at), n - 1, n // 2] = np.nan
    B = Mx.from_mats(Bm)
    W, X, info = run(n, A, B)
    for p, k in enumerate(at):
        assert info[p] == n + k + 1
        assert np.isnan(W[p]).all() and np.isnan(X[p]).all()
    assert info[len(at)] == (n + 1 if n // 2 == n - 1 else 2 * n)
    ok = [len(at) + 1]
    Wr, Xr, ir = oracle_mod.hegv(A[ok], B[ok], n, nthreads=1)
    assert (ir == 0).all()
    check(A[ok], B[ok], W[ok], X[ok], info[ok], Wr, Xr, n)
