"""A zero pivot is refused.  One front whose matrix has a zero column: every
candidate of that column is an exact zero when its turn comes (an update
subtracts multiples of the pivot row's own zero), so that the factorization ends
with LFSOLVE_ERR_SINGULAR and names the position, in one panel block and in a
cluster, in the first column, inside a panel and in the last.  The solver
factors the full matrix afterwards."""

from __future__ import annotations

import pytest

from lithofem_b200.solver import C64, C128
from tests.test_gpu_lu_clusters import one_front, residuals
from tests.test_gpu_sweeps import GATE

pytestmark = pytest.mark.gpu
ERR_SINGULAR = 4


@pytest.mark.parametrize("prec", [C64, C128], ids=["c64", "c128"])
@pytest.mark.parametrize("n", [1, 33, 300, 1300])
def test_zero_column(n, prec):
    lu, A, gen = one_front(n)
    for j in sorted({0, min(45, n - 1), n - 1}):
        S = A.clone()
        S[:, j] = 0.0
        assert not lu.FactorDevice(S.data_ptr(), prec)
        assert lu.last_error[0] == ERR_SINGULAR, lu.last_error
        assert f"zero pivot at position {j + 1} of {n}" in lu.last_error[1]
    assert lu.FactorDevice(A.data_ptr(), prec), lu.last_error
    assert max(residuals(lu, A, gen)) <= GATE[prec]
    lu.Release()


@pytest.mark.parametrize("prec", [C64, C128], ids=["c64", "c128"])
def test_zero_column_on_the_library_path(prec, monkeypatch):
    """Pivot blocks beyond the panel kernel's rows."""
    monkeypatch.setenv("LFSOLVE_LU_MAX", "40")
    lu, A, gen = one_front(70)
    A[:, 50] = 0.0
    assert not lu.FactorDevice(A.data_ptr(), prec)
    assert lu.last_error[0] == ERR_SINGULAR, lu.last_error
    lu.Release()
