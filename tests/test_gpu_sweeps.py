"""The triangular sweeps and the pivot blocks' LU at the edges of their steps
(256 and 32 pivots), links, panel blocks (640 rows in complex64, 320 in
complex128, more in a cluster) and chunks, on synthetic two-element meshes:
the separator's front has s pivots, each leaf's a pivots and s update rows,
so a and s set every size.  Reference: a dense complex128 solve of the same
matrix.  The matrix is dominated by one entry a row (condition number below
10), so the error of a backward stable solve is a small multiple of the unit
roundoff times the front size: 1e-12 covers complex128 (2^-53) and
1e-3 ... 1e-4 complex64 (2^-24) with n up to 2,900; the gates are 1e-11 and
5e-4.  The dominant entries sit on the diagonal, or (shuffled) at a random
permutation of each front's pivots, so that every pivot is an interchange."""

from __future__ import annotations

import ctypes as ct

import numpy as np
import pytest

from lithofem_b200 import solver
from lithofem_b200.solver import C64, C128, DirectSolver

pytestmark = pytest.mark.gpu
GATE = {C64: 5e-4, C128: 1e-11}


def two_elements(a: int, s: int, seed: int, shuffled: bool = False):
    """(solver analysed for the mesh, dense A): element 0 owns DOFs [0, a + s),
    element 1 owns [a, 2 a + s)."""
    nd, n = a + s, 2 * a + s
    dof = np.concatenate([np.arange(nd), np.arange(a, n)]).astype(np.int32)
    mask = np.zeros((n, n), dtype=bool)
    mask[:nd, :nd] = True
    mask[a:, a:] = True
    rng = np.random.default_rng(seed)
    A = np.where(mask, rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)), 0)
    at = np.arange(n)
    if shuffled:
        for own in (at[:a], at[a:nd], at[nd:]):
            own[:] = rng.permutation(own)
    A[np.arange(n), at] += 6.0 * np.sqrt(n) * np.exp(2j * np.pi * rng.random(n))
    J = np.nonzero(mask)[1].astype(np.int32)
    I = np.concatenate([[0], np.cumsum(mask.sum(1))]).astype(np.int32)
    cen = np.array([[0.0, 0.0, 0.0], [1.0, 0.0, 0.0]])
    sv = DirectSolver(0)
    ip = solver._ip
    assert sv._check(solver.lib().lfsolve_analyze(
        sv._s, n, ip(I), ip(J), len(J), 2, nd, ip(dof), cen.ctypes.data_as(ct.POINTER(ct.c_double)),
        None, 0, 1)), sv.last_error
    return sv, A, A[mask]


@pytest.mark.parametrize("prec", [C64, C128], ids=["c64", "c128"])
@pytest.mark.parametrize("a,s", [(1, 1), (31, 33), (32, 32), (33, 95), (65, 96), (255, 257),
                                 (256, 256), (257, 1), (1, 300), (513, 255), (511, 544)])
def test_sweeps_match_a_dense_solve(a, s, prec):
    check(*two_elements(a, s, seed=1000 * a + s), a, s, prec, (1, 2, 3))


@pytest.mark.parametrize("prec", [C64, C128], ids=["c64", "c128"])
@pytest.mark.parametrize("a,s", [(31, 2), (33, 40), (320, 64), (321, 640), (641, 31), (1290, 300)])
def test_lu_with_interchanges(a, s, prec):
    check(*two_elements(a, s, seed=7 * a + s, shuffled=True), a, s, prec, (1,))


@pytest.mark.parametrize("prec", [C64, C128], ids=["c64", "c128"])
def test_pivot_blocks_beyond_the_panel(prec, monkeypatch):
    """The library path of pivot blocks too large for the panel kernel."""
    monkeypatch.setenv("LFSOLVE_LU_MAX", "40")
    check(*two_elements(70, 33, seed=3, shuffled=True), 70, 33, prec, (1,))


@pytest.mark.parametrize("batch_min", ["1", "1000"], ids=["batched", "per-front"])
@pytest.mark.parametrize("a,s", [(16, 16), (64, 65), (65, 64), (130, 70), (600, 49)])
def test_split_products(a, s, batch_min, monkeypatch):
    """The update blocks' leaves of 64 pivots and split TF32 products, forced
    on small fronts (2^-22 a product: inside the complex64 gate)."""
    monkeypatch.setenv("LFSOLVE_TF32X3_MIN", "1")
    monkeypatch.setenv("LFSOLVE_BATCH_MIN", batch_min)
    check(*two_elements(a, s, seed=5 * a + s, shuffled=True), a, s, C64, (1,))


def check(sv, A, vals, a, s, prec, columns):
    import torch
    n = len(A)
    v = torch.from_numpy(vals).cuda()
    assert sv.FactorDevice(v.data_ptr(), prec), sv.last_error
    assert sorted(set(sv.Fronts()["k"])) == sorted({a, s})
    rng = np.random.default_rng(n)
    for nrhs in columns:
        B = rng.standard_normal((nrhs, n)) + 1j * rng.standard_normal((nrhs, n))
        b = torch.from_numpy(B).cuda()
        x = torch.empty_like(b)
        for transpose, M in ((False, A), (True, A.T)):
            assert sv.Backsolve(nrhs, b.data_ptr(), x.data_ptr(), transpose), sv.last_error
            want = np.linalg.solve(M, B.T).T
            err = np.linalg.norm(x.cpu().numpy() - want) / np.linalg.norm(want)
            assert err <= GATE[prec], (nrhs, transpose, err)
    sv.Release()
