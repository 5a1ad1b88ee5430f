"""The pivot blocks' LU in clusters of 2 to 16 blocks (more than 640, 1,280,
2,560 and 5,120 rows in complex64, half of that in complex128): one front per
mesh, its dominant entries at a random permutation of the rows, so that every
pivot row comes from another block, and a row lost between blocks leaves a
pivot six square roots of n too small.  Reference: the residual of a dense
complex128 product with the same matrix, at the gates of
tests/test_gpu_sweeps.py."""

from __future__ import annotations

import ctypes as ct

import numpy as np
import pytest

from lithofem_b200 import solver
from lithofem_b200.solver import C64, C128, DirectSolver
from tests.test_gpu_sweeps import GATE

pytestmark = pytest.mark.gpu


def one_front(n: int):
    """(solver analysed for one element of n DOFs, dense A on the device,
    generator)."""
    import torch
    gen = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn(n, n, dtype=torch.complex128, device="cuda", generator=gen)
    at = torch.randperm(n, device="cuda", generator=gen)
    phase = torch.rand(n, dtype=torch.float64, device="cuda", generator=gen)
    A[torch.arange(n, device="cuda"), at] += 6.0 * n ** 0.5 * torch.exp(2j * np.pi * phase)
    lu = DirectSolver(0)
    ip = solver._ip
    I = np.arange(n + 1, dtype=np.int32) * np.int32(n)
    J = np.tile(np.arange(n, dtype=np.int32), n)
    cen = np.zeros(3)
    assert lu._check(solver.lib().lfsolve_analyze(
        lu._s, n, ip(I), ip(J), n * n, 1, n, ip(J[:n].copy()),
        cen.ctypes.data_as(ct.POINTER(ct.c_double)), None, 0, 1)), lu.last_error
    assert lu.Fronts()["k"].tolist() == [n]
    return lu, A, gen


def residuals(lu, A, gen):
    """Per transpose: the largest relative residual of two solves."""
    import torch
    n = len(A)
    b = torch.randn(2, n, dtype=torch.complex128, device="cuda", generator=gen)
    x = torch.empty_like(b)
    out = []
    for transpose, M in ((False, A), (True, A.T)):
        assert lu.Backsolve(2, b.data_ptr(), x.data_ptr(), transpose), lu.last_error
        out.append(((b - x @ M.T).norm(dim=1) / b.norm(dim=1)).max().item())
    return out


@pytest.mark.parametrize("prec,n", [(C64, 641), (C64, 1300), (C64, 2561), (C64, 5153),
                                    (C128, 321), (C128, 650), (C128, 1281), (C128, 2577)])
def test_panels_of_a_cluster(prec, n):
    lu, A, gen = one_front(n)
    assert lu.FactorDevice(A.data_ptr(), prec), lu.last_error
    assert max(residuals(lu, A, gen)) <= GATE[prec]
    lu.Release()
