"""The reciprocal pivots' rounding: a diagonal system, x_i = b_i / a_i as one
product with the stored reciprocal.  In units of the unit roundoff u the root
mean square of the relative error is 0.42 for a complex number rounded once
and 0.53 for a complex product; a reciprocal within a rounding or so of exact
makes 0.7 of the two, one that carries the roundings of its scaled formula
(0.9 by itself) 1.05.  Gate: 0.9."""

from __future__ import annotations

import ctypes as ct

import numpy as np
import pytest

from lithofem_b200 import solver
from lithofem_b200.solver import C64, C128, DirectSolver

pytestmark = pytest.mark.gpu
U = {C64: 2.0 ** -24, C128: 2.0 ** -53}


@pytest.mark.parametrize("prec", [C64, C128], ids=["c64", "c128"])
def test_reciprocals_are_rounded_about_once(prec):
    import torch
    n = 2048
    real = np.float32 if prec == C64 else np.float64
    rng = np.random.default_rng(5)
    a, b = (rng.standard_normal((2, n)) + 1j * rng.standard_normal((2, n))).astype(
        np.complex64 if real is np.float32 else np.complex128).astype(np.complex128)
    lu = DirectSolver(0)
    ip = solver._ip
    I = np.arange(n + 1, dtype=np.int32) * np.int32(n)
    J = np.tile(np.arange(n, dtype=np.int32), n)
    cen = np.zeros(3)
    assert lu._check(solver.lib().lfsolve_analyze(
        lu._s, n, ip(I), ip(J), n * n, 1, n, ip(J[:n].copy()),
        cen.ctypes.data_as(ct.POINTER(ct.c_double)), None, 0, 1)), lu.last_error
    vals = torch.diag(torch.from_numpy(a)).cuda().contiguous()
    rhs = torch.from_numpy(b).cuda()
    x = torch.empty_like(rhs)
    assert lu.FactorDevice(vals.data_ptr(), prec), lu.last_error
    for transpose in (False, True):
        assert lu.Backsolve(1, rhs.data_ptr(), x.data_ptr(), transpose), lu.last_error
        want = b.astype(np.clongdouble) / a.astype(np.clongdouble)
        err = np.abs(x.cpu().numpy() - want) / np.abs(want) / U[prec]
        assert float(np.sqrt((err ** 2).mean())) <= 0.9, (transpose, float(np.sqrt((err ** 2).mean())))
    lu.Release()
