"""Eigenvectors of spectra with large clusters: inverse iteration for every vector, then the
Newton-Schulz orthonormalisation (csrc/tridiag.cu), and the QL where that cannot work.

Gates of test_gpu_parity.check (residual and B-orthogonality <= 1e-12, clusters by subspace angle).
The orders are the edges of its 32-row blocks and 16-deep panels and of the QL it falls back to
(in the kernel up to n = 63, the rotation log above).
"""
from __future__ import annotations

import numpy as np
import pytest

from oracle import metrics as Mx
from test_gpu_parity import check, run
from test_gpu_invit_edges import random_unitary

pytestmark = pytest.mark.gpu

NS = (12, 16, 31, 33, 54, 63, 64, 65, 84, 96, 97, 160, 192, 256)


def solve_and_check(oracle_mod, n, lam, seed, batch=3):
    rng = np.random.default_rng(seed)
    Cs = []
    for _ in range(batch):
        Q = random_unitary(rng, n)
        C = (Q * lam) @ Q.conj().T
        Cs.append(0.5 * (C + C.conj().T))
    A = Mx.from_mats(np.array(Cs))
    B = Mx.from_mats(np.broadcast_to(np.eye(n), (batch, n, n)).astype(np.complex128))
    W, X, info = run(n, A, B)
    Wr, Xr, ir = oracle_mod.hegv(A, B, n, nthreads=8)
    assert (ir == 0).all()
    check(A, B, W, X, info, Wr, Xr, n)


@pytest.mark.parametrize("n", NS)
def test_one_large_eigenvalue(oracle_mod, n):
    """All eigenvalues but one within 1e-4 of it: one cluster of n - 1, gaps ~1e-5 ||T||."""
    lam = 1e-5 * np.arange(1, n + 1) * (60.0 / n)
    lam[-1] = 10.0
    solve_and_check(oracle_mod, n, lam, n)


@pytest.mark.parametrize("n", [33, 63, 64, 130])
def test_many_pairs_of_close_eigenvalues(oracle_mod, n):
    """More than 32 (n > 64) or 8-in-a-row close eigenvalues, some 1e-9 apart: several steps."""
    lam = np.linspace(-1.0, 1.0, n)
    half = n // 2
    lam[:half] = -1.0 + 2e-5 * np.arange(half)
    lam[1:half:7] = lam[0:half - 1:7][: len(lam[1:half:7])] + 1e-9
    solve_and_check(oracle_mod, n, lam, 1000 + n)


@pytest.mark.parametrize("n", [24, 63, 64, 100, 200])
def test_exact_multiplicities_go_to_the_ql(oracle_mod, n):
    """Two eigenvalues, each n / 2 times, in a full matrix: no vector of the eigenspaces is determined."""
    lam = np.where(np.arange(n) < n // 2, 1.0, -1.0)
    solve_and_check(oracle_mod, n, lam, 2000 + n, batch=2)
