"""The split products' truncation: tensor cores cut every partial sum off
towards zero, so that a product's error grows with the pivots it runs through
in one piece.  Two leaves of 512 identity pivots and positive F12 and F21 whose
products are all close to one: the separator's matrix is s times the identity
once both products are taken from it, and with x = 1 a common relative error
beta of their entries moves x by 2 beta.

Gate: 64 pivots are 128 real terms, 16 steps of the unit's 8; a step cuts off
at most 2^-23 of the sum so far, half of that on average, of half the final sum
on average: beta = 16 / 4 x 2^-23 = 4.8e-7, so 1e-6 in x; the gate is 2e-6.
One piece of 512 pivots cuts off eight times as much."""

from __future__ import annotations

import ctypes as ct

import numpy as np
import pytest

from lithofem_b200 import solver
from lithofem_b200.solver import C64, DirectSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split", [True, False], ids=["split", "fp32"])
@pytest.mark.parametrize("a,s", [(512, 128), (500, 100)])
def test_products_of_positive_terms(a, s, split, monkeypatch):
    import torch
    monkeypatch.setenv("LFSOLVE_TF32X3", "1" if split else "0")
    monkeypatch.setenv("LFSOLVE_TF32X3_MIN", "1")
    nd, n = a + s, 2 * a + s
    rng = np.random.default_rng(a)
    A = np.zeros((n, n), dtype=complex)
    sep = np.arange(a, nd)
    A[np.ix_(sep, sep)] = s * np.eye(s)
    for own in (np.arange(a), np.arange(nd, n)):
        F12, F21 = rng.uniform(0.5, 1.5, (a, s)), rng.uniform(0.5, 1.5, (s, a)) / a
        A[own, own] = 1.0
        A[np.ix_(own, sep)] = F12.astype(np.float32)
        A[np.ix_(sep, own)] = F21.astype(np.float32)
        A[np.ix_(sep, sep)] += A[np.ix_(sep, own)] @ A[np.ix_(own, sep)]
    mask = np.zeros((n, n), dtype=bool)
    mask[:nd, :nd] = True
    mask[a:, a:] = True
    dof = np.concatenate([np.arange(nd), np.arange(a, n)]).astype(np.int32)
    J = np.nonzero(mask)[1].astype(np.int32)
    I = np.concatenate([[0], np.cumsum(mask.sum(1))]).astype(np.int32)
    cen = np.array([0.0, 0.0, 0.0, 1.0, 0.0, 0.0])
    lu = DirectSolver(0)
    ip = solver._ip
    assert lu._check(solver.lib().lfsolve_analyze(
        lu._s, n, ip(I), ip(J), len(J), 2, nd, ip(dof), cen.ctypes.data_as(ct.POINTER(ct.c_double)),
        None, 0, 1)), lu.last_error
    vals = torch.from_numpy(A[mask]).cuda()
    # b = A 1 with the separator's rows alone nonzero after the leaves
    x0 = np.zeros(n, dtype=complex)
    x0[sep] = 1.0
    for own in (np.arange(a), np.arange(nd, n)):
        x0[own] = -(A[np.ix_(own, sep)].sum(1))
    b = torch.from_numpy(A @ x0).cuda()
    x = torch.empty_like(b)
    assert lu.FactorDevice(vals.data_ptr(), C64), lu.last_error
    assert lu.Backsolve(1, b.data_ptr(), x.data_ptr()), lu.last_error
    assert np.abs(x.cpu().numpy()[sep] - 1.0).max() <= 2e-6
    lu.Release()
