"""The reported shared memory covers every kernel that is launched.

Lower bounds from three kernels' own layouts: the QL chain keeps 2 n doubles a thread (n > 63), the tensor-core
Cholesky the 8 x 8 blocks of L's triangle and of its diagonal's inverses, 72 complex each (n <= 144), the refinement
two complex n x (n + 4) tiles padded to 8 (mixed, n <= 63).
"""
from __future__ import annotations

import pytest

import sbg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [16, 54, 63, 64, 72, 84, 85, 112, 128, 144, 160, 256])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_reported_shared_memory(n, precision):
    if n > sbg.max_n(precision):
        pytest.skip(f"the {precision} form covers n <= {sbg.max_n(precision)}")
    s = sbg.Solver(n, precision=precision)
    need = 0
    if n > 63:
        need = 16 * n * s.schedule["chain_threads"]
    if n <= 144:
        blocks = (n + 7) // 8
        need = max(need, 16 * 72 * (blocks * (blocks + 1) // 2 + blocks))
    if n <= 63 and precision == "mixed":
        padded = (n + 7) // 8 * 8
        need = max(need, 2 * 16 * padded * (padded + 4))
    assert need <= s.shared_mem_bytes <= 232448
    s.close()


def test_fixed_n54_reports():
    d = sbg.fixed_n54_introspection()
    whole = d["geneig_full_n54_batched_shared_mem_bytes"]
    assert whole == sbg.Solver(54).shared_mem_bytes
    assert 0 < d["geneig_reduce_eig_n54_heev_smem_bytes"] <= whole
    assert 0 < d["geneig_reduce_eig_n54_chol_smem_bytes"] <= whole
