"""Backward stability of the triangles: pivot blocks whose 32 x 32 diagonal
blocks have inverses of size 2^30 (unit triangles of -1 times random pivots),
lower ones (they become L11, no interchange wins a tie) and upper ones (they
become U11), in the sweeps alone (one front) and in the update blocks too (two
leaves whose F12 and F21 are products with the triangle, so that U12, L21 and
the separator's front are of ordinary size).

Gate: the backward error ||b - A x|| / (||A|| ||x|| + ||b||) (infinity norms,
the residual in complex128) of substitution is below n u for n rows and unit
roundoff u; 4 n u leaves room for complex arithmetic.  A product with an
explicit inverse errs by up to 2^30 u."""

from __future__ import annotations

import ctypes as ct

import numpy as np
import pytest

from lithofem_b200 import solver
from lithofem_b200.solver import C64, C128, DirectSolver

pytestmark = pytest.mark.gpu
U = {C64: 2.0 ** -24, C128: 2.0 ** -53}


def triangle(a: int, lower: bool, rng) -> np.ndarray:
    T = np.zeros((a, a), dtype=complex)
    for j in range(0, a, 32):
        n = min(32, a - j)
        B = np.eye(n) - (np.tril if lower else np.triu)(np.ones((n, n)), -1 if lower else 1)
        d = rng.uniform(1.0, 2.0, n) * np.exp(2j * np.pi * rng.random(n))
        T[j:j + n, j:j + n] = B * d if lower else d[:, None] * B
    return T


def system(a: int, s: int, lower: bool, seed: int):
    """(A, element DOFs): one element of a DOFs (s = 0), or two of a + s that
    share s; the matrix's rows and columns in the elements' order."""
    rng = np.random.default_rng(seed)
    T = triangle(a, lower, rng)
    if s == 0:
        return T, np.arange(a)[None]
    n = 2 * a + s
    A = np.zeros((n, n), dtype=complex)
    own = [np.arange(a), np.arange(a + s, n)]
    sep = np.arange(a, a + s)
    A[np.ix_(sep, sep)] = 8.0 * np.eye(s)
    for p in own:
        G, H = (rng.standard_normal((2, a, s)) + 1j * rng.standard_normal((2, a, s))) / np.sqrt(8 * a)
        A[np.ix_(p, p)] = T
        A[np.ix_(p, sep)] = T @ G
        A[np.ix_(sep, p)] = H.T @ T
        A[np.ix_(sep, sep)] += H.T @ T @ G
    return A, np.stack([np.r_[own[0], sep], np.r_[sep, own[1]]])


@pytest.mark.parametrize("prec", [C64, C128], ids=["c64", "c128"])
@pytest.mark.parametrize("lower", [True, False], ids=["lower", "upper"])
@pytest.mark.parametrize("a,s", [(32, 0), (45, 0), (300, 0), (32, 16), (64, 40), (100, 70)])
def test_triangles_are_backward_stable(a, s, lower, prec):
    import torch
    A, dof = system(a, s, lower, seed=a + s)
    n, (ne, nd) = len(A), dof.shape
    mask = np.zeros((n, n), dtype=bool)
    for d in dof:
        mask[np.ix_(d, d)] = True
    J = np.nonzero(mask)[1].astype(np.int32)
    I = np.concatenate([[0], np.cumsum(mask.sum(1))]).astype(np.int32)
    lu = DirectSolver(0)
    ip = solver._ip
    dof = np.ascontiguousarray(dof, dtype=np.int32)
    cen = np.zeros((ne, 3))
    cen[:, 0] = np.arange(ne)
    assert lu._check(solver.lib().lfsolve_analyze(
        lu._s, n, ip(I), ip(J), len(J), ne, nd, ip(dof), cen.ctypes.data_as(ct.POINTER(ct.c_double)),
        None, 0, 1)), lu.last_error
    vals = torch.from_numpy(A[mask]).cuda()
    assert lu.FactorDevice(vals.data_ptr(), prec), lu.last_error
    rng = np.random.default_rng(n)
    x0 = rng.standard_normal((2, n)) + 1j * rng.standard_normal((2, n))
    for nrhs in (1, 2):
        for transpose, M in ((False, A), (True, A.T)):
            B = np.ascontiguousarray(x0[:nrhs] @ M.T)
            b = torch.from_numpy(B).cuda()
            x = torch.empty_like(b)
            assert lu.Backsolve(nrhs, b.data_ptr(), x.data_ptr(), transpose), lu.last_error
            X = x.cpu().numpy()
            norm = np.abs(M).sum(1).max() * np.abs(X).max(1) + np.abs(B).max(1)
            err = (np.abs(B - X @ M.T).max(1) / norm).max()
            assert err <= 4 * n * U[prec], (nrhs, transpose, err / U[prec])
    lu.Release()
