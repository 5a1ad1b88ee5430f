"""The sweeps at the front counts where their kernels change: trees of many
like leaves under one separator, so that a depth has 2, 32 or 64
fronts whose pivots need more than one step of 256, at one and two columns, as
they are and transposed.  Reference: the residual of a dense complex128 product
with the same matrix (dominated rows, condition number below 10: 1e-11 in
complex128, 5e-4 in complex64, the gates of tests/test_gpu_sweeps.py)."""

from __future__ import annotations

import numpy as np
import pytest

from lithofem_b200.solver import C64, C128, DirectSolver

pytestmark = pytest.mark.gpu
GATE = {C64: 5e-4, C128: 1e-11}


def comb(leaves: int, a: int, s: int, seed: int):
    """`leaves` elements of a own DOFs each and s DOFs that all share: the
    separator is the root, a leaf an element (bisection along x)."""
    nd, n = a + s, leaves * a + s
    dof = np.array([np.r_[e * a:(e + 1) * a, leaves * a:n] for e in range(leaves)], dtype=np.int32)
    rng = np.random.default_rng(seed)
    rows, cols = [], []
    for e in range(leaves):
        i, j = np.meshgrid(dof[e], dof[e], indexing="ij")
        rows.append(i.ravel())
        cols.append(j.ravel())
    key = np.unique(np.concatenate(rows).astype(np.int64) * n + np.concatenate(cols))
    i, j = key // n, key % n
    v = (rng.standard_normal(len(key)) + 1j * rng.standard_normal(len(key))) / np.sqrt(n)
    v[i == j] += 8.0
    I = np.zeros(n + 1, dtype=np.int32)
    np.cumsum(np.bincount(i, minlength=n), out=I[1:])
    return n, nd, dof, I, j.astype(np.int32), v


@pytest.mark.parametrize("prec", [C64, C128], ids=["c64", "c128"])
@pytest.mark.parametrize("leaves,a,s", [(2, 300, 520), (33, 290, 40), (64, 270, 300)])
def test_depths(leaves, a, s, prec):
    import ctypes as ct

    import torch

    from lithofem_b200 import solver
    n, nd, dof, I, J, v = comb(leaves, a, s, seed=leaves)
    cen = np.zeros((leaves, 3))
    cen[:, 0] = np.arange(leaves)
    lu = DirectSolver(0)
    ip = lambda x: x.ctypes.data_as(ct.POINTER(ct.c_int))
    ess = np.zeros(1, dtype=np.int32)
    rc = solver.lib().lfsolve_analyze(
        lu._s, n, ip(I), ip(J), len(J), leaves, nd, ip(np.ascontiguousarray(dof.reshape(-1))),
        np.ascontiguousarray(cen.reshape(-1)).ctypes.data_as(ct.POINTER(ct.c_double)), ip(ess), 0, 1)
    assert rc == 0, solver.lib().lfsolve_last_error()
    vals = torch.from_numpy(v).cuda()
    assert lu.FactorDevice(vals.data_ptr(), prec), lu.last_error
    import scipy.sparse as sp
    A = sp.csr_matrix((v, J, I), shape=(n, n))
    rng = np.random.default_rng(1)
    for nrhs in (1, 2):
        b = rng.standard_normal((nrhs, n)) + 1j * rng.standard_normal((nrhs, n))
        bd = torch.from_numpy(b).cuda()
        for transpose in (False, True):
            x = torch.zeros_like(bd)
            assert lu.Backsolve(nrhs, bd.data_ptr(), x.data_ptr(), transpose), lu.last_error
            y = (A.T if transpose else A) @ x.cpu().numpy().T
            res = np.abs(y.T - b).max() / np.abs(b).max()
            assert res < GATE[prec], (nrhs, transpose, res)
    lu.Release()
