"""The one-kernel eigensolve of the smallest orders (csrc/tridiag.cu, k_tridiag_tiny) and the order above it.

Bounds as in test_gpu_tridiag_values (64 n eps ||A||) and test_gpu_parity (vectors).
"""
from __future__ import annotations

import numpy as np
import pytest
import torch

import sbg
from oracle import metrics as Mx
from test_gpu_parity import TOL, run

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def hermitian(n, batch, seed):
    rng = np.random.default_rng(seed)
    G = rng.normal(size=(batch, n, n)) + 1j * rng.normal(size=(batch, n, n))
    return G + G.conj().transpose(0, 2, 1)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5])
def test_against_lapack(n, precision):
    A = hermitian(n, 40, n)
    A[30:35] = np.eye(n) * 2.5                        # every eigenvalue the same
    A[35:] = np.diag(np.arange(n) - 1.5)              # T diagonal
    B = np.eye(n) + 0.1 * hermitian(n, 40, 50 + n) / n
    W, X, info = run(n, Mx.from_mats(A), Mx.from_mats(B), precision)
    L = np.linalg.inv(np.linalg.cholesky(B))
    ref = np.linalg.eigvalsh(L @ A @ L.conj().transpose(0, 2, 1))
    assert (info == 0).all() and (np.diff(W, axis=1) >= 0).all()
    assert (np.abs(W - ref).max(axis=1) <= 64 * n * EPS * np.abs(ref).max(axis=1)).all()
    Xm = X.reshape(-1, n, n).transpose(0, 2, 1)
    assert np.abs(Xm.conj().transpose(0, 2, 1) @ B @ Xm - np.eye(n)).max() <= TOL
    R = A @ Xm - (B @ Xm) * W[:, None, :]
    assert (np.linalg.norm(R, axis=(1, 2)) <= TOL * np.linalg.norm(A, axis=(1, 2)) * np.linalg.norm(Xm, axis=(1, 2))).all()


@pytest.mark.parametrize("n", [2, 3, 4, 5])
def test_info_codes(n):
    """B not positive definite, a NaN, and ordinary pairs beside them."""
    A = hermitian(n, 4, 9)
    B = np.broadcast_to(np.eye(n), A.shape).astype(np.complex128).copy()
    B[1, 1, 1] = -1.0
    A[2, 0, 0] = np.nan
    W, X, info = run(n, Mx.from_mats(A), Mx.from_mats(B))
    assert list(info) == [0, n + 2, n - 1, 0]
    assert np.isnan(W[1:3]).all() and np.isnan(X[1:3]).all()
    for p in (0, 3):
        ref = np.linalg.eigvalsh(A[p])
        assert np.abs(W[p] - ref).max() <= 64 * n * EPS * np.abs(ref).max()


@pytest.mark.parametrize("n,launches", [(1, 1), (2, 1), (4, 1), (5, 3)])
def test_eigensolve_launches(n, launches):
    s = sbg.Solver(n)
    s.enable_stage_timing()
    A = torch.eye(n, dtype=torch.complex128, device="cuda").reshape(1, -1).contiguous()
    W = torch.empty((1, n), dtype=torch.float64, device="cuda")
    s.launch(A, A, W, torch.empty_like(A), torch.empty(1, dtype=torch.int32, device="cuda"))
    assert s.read_stage_times()["eig"][1] == launches
    s.close()
