"""Inverse iteration on close eigenvalues around the overlap (1e-6, eigenvalues ~1e-10 ||T|| apart) where
the kernel turns from one Gram-Schmidt step over vectors computed alone to computing the members again.

Gates of test_gpu_parity.check (residual and B-orthogonality <= 1e-12, clusters by subspace angle): both
sides keep a vector's residual at ~1e-14 ||T|| and its overlaps at ~1e-15.  The orders are the edges of
the kernel's batches of lanes (1, 2, 3 and 4 batches).
"""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_tridiag_ortho import solve_and_check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gap", [3e-12, 3e-11, 1e-10, 3e-10, 3e-9, 1e-7])
@pytest.mark.parametrize("n", [4, 32, 33, 54, 65, 97])
def test_close_triples(oracle_mod, n, gap):
    lam = np.linspace(-1.0, 1.0, n)
    for s in range(0, n - 2, max(4, n // 4)):
        lam[s + 1], lam[s + 2] = lam[s] + gap, lam[s] + 3.0 * gap
    solve_and_check(oracle_mod, n, np.sort(lam), n, batch=4)
