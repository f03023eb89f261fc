"""The tensor-core back-transform (csrc/back_dmma.cu) at the edges of its 8-column tiles.

Every remainder of 8 and both ends of each tile count's range, against zhegv under the gates of
test_gpu_parity.check, for the whole solve (Q and L^{-H} in one launch) and for the mixed form (Q,
then L^{-H} after the refinement); pairs whose B is not positive definite give NaN and leave their
neighbours alone.
"""
from __future__ import annotations

import numpy as np
import pytest

from oracle import metrics as Mx
from test_gpu_hetrd_shapes import pair
from test_gpu_parity import check, run

pytestmark = pytest.mark.gpu

EDGES = sorted({8 * t + r for t in range(0, 13) for r in (0, 1)} | set(range(49, 57)) | {7, 87, 95}) [1:]


# the streamed form: its tile counts (two apart), a last tile of one row, one and two passes over the panels
STREAM = (98, 104, 105, 112, 113, 127, 136, 143, 153, 168, 177, 185, 191, 192, 193)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", EDGES + list(STREAM))
def test_every_tile_count(oracle_mod, n, precision):
    rng = np.random.default_rng(500 + n)
    ps = [pair(rng, n) for _ in range(3)]
    A = Mx.from_mats(np.array([p[0] for p in ps]))
    Bm = np.array([p[1] for p in ps]).astype(np.complex128)
    Wr, Xr, ir = oracle_mod.hegv(A, Mx.from_mats(Bm), n, nthreads=4)
    assert (ir == 0).all()
    bad = Bm.copy()
    bad[1] = -bad[1]
    W, X, info = run(n, A, Mx.from_mats(bad), precision)
    assert info[1] == n + 1 and np.isnan(X[1]).all() and np.isnan(W[1]).all()
    ok = [0, 2]
    check(A[ok], Mx.from_mats(Bm[ok]), W[ok], X[ok], info[ok], Wr[ok], Xr[ok], n)
