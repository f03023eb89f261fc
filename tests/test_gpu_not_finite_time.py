"""A pair whose tridiagonal is not finite is given up at once: NaN out, info = n - 1, and no time spent on QL
sweeps that cannot converge (30 n of them by one thread: 8 s for one pair of n = 256).

The bound on time is a factor of 20 on a solve of finite pairs; the sweeps took 30 (n = 54) to 250 times that.
"""
from __future__ import annotations

import numpy as np
import pytest
import torch

import sbg
from oracle import metrics as Mx

pytestmark = pytest.mark.gpu


# the warp QL (n <= 63), the rotation log above, every Householder kernel
@pytest.mark.parametrize("n", [32, 54, 63, 64, 72, 96, 128, 160, 256])
def test_not_finite_costs_no_sweeps(n):
    rng = np.random.default_rng(n)
    G = rng.normal(size=(4, n, n)) + 1j * rng.normal(size=(4, n, n))
    A = G + G.conj().transpose(0, 2, 1)
    bad = A.copy()
    bad[1, 0, 0] = np.nan
    bad[2, n - 1, n - 1] = np.inf
    bad[3, n - 1, 0] = bad[3, 0, n - 1] = np.nan
    s = sbg.Solver(n)
    dB = torch.as_tensor(Mx.from_mats(np.broadcast_to(np.eye(n), A.shape).astype(np.complex128))).cuda()
    ms = {}
    for name, M in (("finite", A), ("bad", bad)):
        dA = torch.as_tensor(Mx.from_mats(M)).cuda()
        W = torch.empty((4, n), dtype=torch.float64, device="cuda")
        X = torch.empty_like(dA)
        info = torch.full((4,), -7, dtype=torch.int32, device="cuda")
        best = np.inf
        for _ in range(3):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            s.launch(dA, dB, W, X, info)
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b))
        ms[name] = best
    s.close()
    W, X, info = W.cpu().numpy(), X.cpu().numpy(), info.cpu().numpy()
    assert list(info) == [0, n - 1, n - 1, n - 1]
    assert np.isfinite(W[0]).all() and np.isfinite(X[0]).all()
    assert np.isnan(W[1:]).all() and np.isnan(X[1:]).all()
    assert np.abs(W[0] - np.linalg.eigvalsh(A[0])).max() <= 64 * n * 2.0 ** -53 * np.abs(W[0]).max()
    assert ms["bad"] <= 20 * ms["finite"], ms
