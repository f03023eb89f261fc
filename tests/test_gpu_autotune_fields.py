"""The autotuner changes no field that it cannot have measured: every launch of its pairs is the same for all values
of the remaining fields, so what it keeps is the built-in schedule and what the caller asked for."""
from __future__ import annotations

import pytest

import sbg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [12, 40, 54, 72, 96])
def test_only_what_was_asked_for(n, precision):
    builtin = sbg.Solver(n, precision=precision).schedule
    s = sbg.Solver(n, precision=precision, tuning="autotune", cache="none")
    assert s.autotune_sweep_ran and s.schedule == builtin
    s.close()
    asked = sbg.Solver(n, precision=precision, tuning="autotune", cache="none", block_dim=128, batches_per_block=1)
    field = "pairs_per_cta" if n <= 65 else "ql_warps"
    assert asked.autotune_sweep_ran and asked.schedule == dict(builtin, hetrd_threads=128, **{field: 1})
    asked.close()
