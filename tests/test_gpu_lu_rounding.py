"""Rounding errors of the pivot blocks' LU: the residuals of one dense front
(tests/test_gpu_lu_clusters.py) at the sizes of one panel block and of clusters.
The matrix's dominant entries are six times the norm of the rest of their row,
so that nothing grows and the rounding errors of a row stay a small multiple of
the unit roundoff u of its right-hand side, as long as an update's terms are
summed before they meet the dominant entry: the gates are 17 u (1e-6 and
2e-15)."""

from __future__ import annotations

import pytest

from lithofem_b200.solver import C64, C128
from tests.test_gpu_lu_clusters import one_front, residuals

pytestmark = pytest.mark.gpu
GATE = {C64: 1e-6, C128: 2e-15}


@pytest.mark.parametrize("prec,n", [(C64, 641), (C64, 1300), (C64, 2561), (C64, 5153),
                                    (C128, 321), (C128, 650), (C128, 1281), (C128, 2577)])
def test_residuals_of_a_dense_front(prec, n):
    lu, A, gen = one_front(n)
    assert lu.FactorDevice(A.data_ptr(), prec), lu.last_error
    assert max(residuals(lu, A, gen)) <= GATE[prec]
    lu.Release()
