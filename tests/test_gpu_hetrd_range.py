"""Householder columns whose squared norm leaves the normal range, in an otherwise ordinary matrix.

A column of norm 1e-154 to 1e-162 has a subnormal or vanishing square, one of 1e153 and more an
overflowing one; LAPACK's zlarfg rescales such columns.  B = I, so that C = A.  Bounds: Householder's
backward error is O(n eps) ||A|| (64 n eps ||A|| on the eigenvalues, as in test_gpu_tridiag_values); the
vectors are gated as in test_gpu_parity.
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
# one and two to five rows per lane, one to eight warps, and the packed triangle above n = 144
NS = [3, 8, 24, 32, 47, 54, 64, 72, 96, 128, 144, 160, 200]


def hermitian(n, batch, seed):
    rng = np.random.default_rng(seed)
    G = rng.normal(size=(batch, n, n)) + 1j * rng.normal(size=(batch, n, n))
    return G + G.conj().transpose(0, 2, 1)


def with_column(A, k, t):
    """Column k's entries below the diagonal replaced by a single t two rows below it."""
    A = A.copy()
    A[:, k + 1:, k] = 0.0
    A[:, k, k + 1:] = 0.0
    A[:, k + 2, k] = t
    A[:, k, k + 2] = np.conj(t)
    return A


def check(A, W, X, info, scale=1.0):
    """A in ordinary range; the pair solved was A * scale."""
    b, n, _ = A.shape
    assert (info == 0).all(), info
    ref = np.linalg.eigvalsh(A)
    assert np.abs(W / scale - ref).max() <= 64 * n * EPS * np.abs(ref).max()
    Xm = X.reshape(b, n, n).transpose(0, 2, 1)
    assert np.abs(Xm.conj().transpose(0, 2, 1) @ Xm - np.eye(n)).max() <= TOL
    R = A @ Xm - Xm * (W / scale)[:, None, :]
    assert np.linalg.norm(R, axis=(1, 2)).max() <= TOL * np.linalg.norm(A, axis=(1, 2)).min()


@pytest.mark.parametrize("n", NS)
@pytest.mark.parametrize("t", [1e-153, 1e-154, 1e-157j, 1e-161, 1e-170, 1e-300j])
def test_tiny_column(n, t):
    A = with_column(hermitian(n, 2, n), 0, t)
    W, X, info = run(n, Mx.from_mats(A), Mx.from_mats(np.broadcast_to(np.eye(n), A.shape).astype(np.complex128)))
    check(A, W, X, info)


@pytest.mark.parametrize("n", NS)
@pytest.mark.parametrize("scale", [1e-160, 1e-154, 1e152, 1e153])
def test_whole_matrix_at_the_edge(n, scale):
    A = hermitian(n, 2, 100 + n)
    W, X, info = run(n, Mx.from_mats(A * scale), Mx.from_mats(np.broadcast_to(np.eye(n), A.shape).astype(np.complex128)))
    check(A, W, X, info, scale)



def test_staged_finish():
    """The reduced matrix in the caller's own (read-only) buffer."""
    n = 54
    A = with_column(hermitian(n, 3, 7), 0, 1e-157)
    M = torch.as_tensor(Mx.from_mats(np.tril(A))).cuda()
    L = torch.as_tensor(Mx.from_mats(np.broadcast_to(np.eye(n), A.shape).astype(np.complex128))).cuda()
    kept = M.clone()
    W = torch.empty((3, n), dtype=torch.float64, device="cuda")
    U = torch.empty_like(M)
    info = torch.full((3,), -7, dtype=torch.int32, device="cuda")
    sbg.finish_n54(L, M, W, U, info, 3)
    torch.cuda.synchronize()
    check(A, W.cpu().numpy(), U.cpu().numpy(), info.cpu().numpy())
    assert torch.equal(M, kept)
