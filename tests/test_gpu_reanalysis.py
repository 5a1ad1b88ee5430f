"""One solver analysed for one mesh after another: small, then larger (the
factors, pivot and status arrays of the first must not be written by the
second), then smaller with more columns (the refined solve's scratch).  Between
an analysis and its factorization a solve is refused.  Reference: dense
complex128 solves (the systems and gates of tests/test_gpu_sweeps.py)."""

from __future__ import annotations

import ctypes as ct

import numpy as np
import pytest

from lithofem_b200 import solver
from lithofem_b200.solver import C64, C128, DirectSolver
from tests.test_gpu_sweeps import GATE

pytestmark = pytest.mark.gpu
ERR_STATE = 3


def analyse(lu, a: int, s: int):
    """Two elements that share s DOFs, a more each; (dense A, I, J)."""
    nd, n = a + s, 2 * a + s
    rng = np.random.default_rng(n)
    mask = np.zeros((n, n), dtype=bool)
    mask[:nd, :nd] = True
    mask[a:, a:] = True
    A = np.where(mask, rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)), 0)
    A[np.arange(n), np.arange(n)] += 6.0 * np.sqrt(n)
    dof = np.concatenate([np.arange(nd), np.arange(a, n)]).astype(np.int32)
    J = np.nonzero(mask)[1].astype(np.int32)
    I = np.concatenate([[0], np.cumsum(mask.sum(1))]).astype(np.int32)
    cen = np.array([0.0, 0.0, 0.0, 1.0, 0.0, 0.0])
    ip = solver._ip
    assert lu._check(solver.lib().lfsolve_analyze(
        lu._s, n, ip(I), ip(J), len(J), 2, nd, ip(dof), cen.ctypes.data_as(ct.POINTER(ct.c_double)),
        None, 0, 1)), lu.last_error
    return A, I, J, A[mask]


@pytest.mark.parametrize("prec", [C64, C128], ids=["c64", "c128"])
def test_meshes_one_after_another(prec):
    import torch
    L = solver.lib()
    lu = DirectSolver(0)
    for a, s, nrhs in ((20, 10, 1), (400, 130, 2), (30, 20, 40)):
        A, I, J, v = analyse(lu, a, s)
        n = len(A)
        rng = np.random.default_rng(nrhs)
        B = rng.standard_normal((nrhs, n)) + 1j * rng.standard_normal((nrhs, n))
        b = torch.from_numpy(B).cuda()
        x = torch.empty_like(b)
        assert not lu.Backsolve(nrhs, b.data_ptr(), x.data_ptr())
        assert lu.last_error[0] == ERR_STATE
        vals = torch.from_numpy(v).cuda()
        dI, dJ = torch.from_numpy(I).cuda(), torch.from_numpy(J).cuda()
        P = ct.c_void_p
        rel, it = (ct.c_double * nrhs)(), ct.c_int(0)
        refined = lambda: L.lfsolve_solve_refined(
            lu._s, P(dI.data_ptr()), P(dJ.data_ptr()), P(vals.data_ptr()), nrhs, P(b.data_ptr()),
            P(x.data_ptr()), 0, 1e-12, 5, rel, ct.byref(it))
        assert refined() == ERR_STATE
        want = np.linalg.solve(A, B.T).T
        for _ in range(2):
            assert lu.FactorDevice(vals.data_ptr(), prec), lu.last_error
            assert lu.Backsolve(nrhs, b.data_ptr(), x.data_ptr()), lu.last_error
            assert np.linalg.norm(x.cpu().numpy() - want) <= GATE[prec] * np.linalg.norm(want)
        assert refined() == 0, L.lfsolve_last_error()
        assert max(rel) <= 1e-12
        assert np.linalg.norm(x.cpu().numpy() - want) <= 1e-11 * np.linalg.norm(want)
    lu.Release()
