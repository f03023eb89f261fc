"""Edges of the bisection eigenvalue kernel (csrc/tridiag.cu), through the solver.

The Sturm counts are exact for a T perturbed by a few eps per entry and the Householder
tridiagonalisation adds a backward error of O(n eps) ||A||: 64 n eps ||A|| bounds both.
"""
from __future__ import annotations

import numpy as np
import pytest

from oracle import metrics as Mx
from test_gpu_parity import run

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def hermitian(n, batch, seed, scale=1.0):
    rng = np.random.default_rng(seed)
    G = rng.normal(size=(batch, n, n)) + 1j * rng.normal(size=(batch, n, n))
    return scale * (G + G.conj().transpose(0, 2, 1))


def eye(n, batch):
    return Mx.from_mats(np.broadcast_to(np.eye(n), (batch, n, n)).astype(np.complex128))


# one and two eigenvalues per thread, one to four warps, remainders of the 8-row blocks
@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 31, 32, 33, 54, 63, 64, 65, 96, 127, 128])
def test_against_lapack(n):
    batch = 5
    A = hermitian(n, batch, n)
    W, _, info = run(n, Mx.from_mats(A), eye(n, batch))
    ref = np.linalg.eigvalsh(A)
    assert (info == 0).all() and (np.diff(W, axis=1) >= 0).all()
    assert np.abs(W - ref).max() <= 64 * n * EPS * np.abs(ref).max()


@pytest.mark.parametrize("scale", [1e-140, 1e140])
def test_extreme_scales(scale):
    n, batch = 33, 3
    A = hermitian(n, batch, 5)
    W, _, info = run(n, Mx.from_mats(A * scale), eye(n, batch))
    ref = np.linalg.eigvalsh(A)
    assert (info == 0).all()
    assert np.abs(W / scale - ref).max() <= 64 * n * EPS * np.abs(ref).max()


@pytest.mark.parametrize("n", [1, 5, 32, 40, 100])
def test_diagonal_is_exact(n):
    """T diagonal: its entries sorted, zeros, repeats and tiny values included."""
    d = np.random.default_rng(n).normal(size=n)
    d[: n // 3] = 0.0
    d[n // 3: n // 2] = 1e-30
    W, _, info = run(n, Mx.from_mats(np.diag(d).astype(np.complex128)[None]), eye(n, 1))
    assert (info == 0).all() and np.array_equal(W[0], np.sort(d))


@pytest.mark.parametrize("n", [12, 54, 100])
def test_not_finite_pair_is_reported_alone(n):
    """A NaN or an infinity in one pair: an info code for it, the others solved."""
    A = hermitian(n, 4, 9)
    ref = np.linalg.eigvalsh(A)
    A[1, 0, 0] = np.nan
    A[2, n - 1, n - 1] = np.inf
    W, _, info = run(n, Mx.from_mats(A), eye(n, 4))
    assert info[0] == 0 and info[3] == 0 and 0 < info[1] <= n and 0 < info[2] <= n
    for p in (0, 3):
        assert np.abs(W[p] - ref[p]).max() <= 64 * n * EPS * np.abs(ref[p]).max()


@pytest.mark.parametrize("n", [21, 41, 63, 101, 255])
def test_pairs_equal_to_the_last_bit(n):
    """Wilkinson's W+: its larger eigenvalues come in pairs that agree to machine precision, so their
    brackets are never isolated; and a T whose eigenvalues spread over ten decades."""
    m = n // 2
    A = np.diag(np.abs(np.arange(n) - m).astype(np.complex128)) + np.diag(np.ones(n - 1), 1) + np.diag(np.ones(n - 1), -1)
    d = 10.0 ** np.linspace(0.0, -10.0, n)
    G = np.diag(d).astype(np.complex128) + np.diag(0.4 * np.sqrt(d[1:] * d[:-1]), 1) + np.diag(0.4 * np.sqrt(d[1:] * d[:-1]), -1)
    P = np.array([A, G])
    W, _, info = run(n, Mx.from_mats(P), eye(n, 2))
    ref = np.linalg.eigvalsh(P)
    assert (info == 0).all() and (np.diff(W, axis=1) >= 0).all()
    assert (np.abs(W - ref).max(axis=1) <= 64 * n * EPS * np.abs(ref).max(axis=1)).all()
