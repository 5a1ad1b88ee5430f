"""The pivot is the largest |re| + |im| in full precision.  Two rows whose
first entries agree in their leading bits (30 bits of a complex128, 20 of a
complex64): with the larger one as pivot the multiplier is below one and the
second column's entry M, the largest finite number, stays as it is; with the
smaller one the multiplier is above one and its product with M overflows.
x = (1, 1) then comes back to the last bits."""

from __future__ import annotations

import ctypes as ct

import numpy as np
import pytest

from lithofem_b200 import solver
from lithofem_b200.solver import C64, C128, DirectSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,bits,M", [(C128, 30, np.finfo(np.float64).max),
                                         (C64, 20, float(np.finfo(np.float32).max))],
                         ids=["c128", "c64"])
@pytest.mark.parametrize("first", [0, 1])
def test_larger_entry_wins_by_its_last_bits(prec, bits, M, first):
    import torch
    big = 1.0 + 2.0 ** -bits
    A = np.zeros((2, 2), dtype=complex)
    A[first] = (1.0, M)
    A[1 - first] = (big, 0.0)
    b = np.zeros(2, dtype=complex)
    b[first], b[1 - first] = M, big
    lu = DirectSolver(0)
    ip = solver._ip
    I = np.array([0, 2, 4], dtype=np.int32)
    J = np.array([0, 1, 0, 1], dtype=np.int32)
    cen = np.zeros(3)
    assert lu._check(solver.lib().lfsolve_analyze(
        lu._s, 2, ip(I), ip(J), 4, 1, 2, ip(J[:2].copy()),
        cen.ctypes.data_as(ct.POINTER(ct.c_double)), None, 0, 1)), lu.last_error
    vals, rhs = torch.from_numpy(A).cuda(), torch.from_numpy(b).cuda()
    x = torch.empty_like(rhs)
    assert lu.FactorDevice(vals.data_ptr(), prec), lu.last_error
    assert lu.Backsolve(1, rhs.data_ptr(), x.data_ptr()), lu.last_error
    eps = np.finfo(np.float64 if prec == C128 else np.float32).eps
    assert np.abs(x.cpu().numpy() - 1.0).max() <= 4 * eps, x
    lu.Release()
