"""What a first solve allocates.  20,000 small leaves under one shared DOF: no
depth splits its first backward product, so that the scratch is the vectors
alone (per right-hand-side column of a pass: the fronts' rows, the pivots, the
right-hand side and the solution), within 16 MB of allocation granules."""

from __future__ import annotations

import ctypes as ct

import numpy as np
import pytest

from lithofem_b200 import solver
from lithofem_b200.solver import C128, DirectSolver
from tests.test_gpu_sweep_depths import comb

pytestmark = pytest.mark.gpu


def test_no_partial_sums_without_parts():
    import torch
    leaves, a, s = 20000, 10, 1
    n, nd, dof, I, J, v = comb(leaves, a, s, seed=1)
    cen = np.zeros((leaves, 3))
    cen[:, 0] = np.arange(leaves)
    ip = solver._ip
    dof = np.ascontiguousarray(dof.reshape(-1))
    vals = torch.from_numpy(v).cuda()
    b = torch.ones(2, n, dtype=torch.complex128, device="cuda")
    x = torch.empty_like(b)
    for _ in range(2):      # the first one loads the kernels
        lu = DirectSolver(0)
        assert lu._check(solver.lib().lfsolve_analyze(
            lu._s, n, ip(I), ip(J), len(J), leaves, nd, ip(dof),
            cen.ctypes.data_as(ct.POINTER(ct.c_double)), None, 0, 1)), lu.last_error
        assert lu.FactorDevice(vals.data_ptr(), C128), lu.last_error
        free = torch.cuda.mem_get_info()[0]
        assert lu.Backsolve(2, b.data_ptr(), x.data_ptr()), lu.last_error
        taken = free - torch.cuda.mem_get_info()[0]
        vectors = 2 * 16 * (int(lu.Fronts()["m"].sum()) + n + 2 * n)
        lu.Release()
    assert taken <= vectors + (16 << 20), (taken, vectors)
