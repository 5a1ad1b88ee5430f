"""Gates at the size of the errors.  The dominated systems of
tests/test_gpu_sweeps.py have condition numbers below 10: an FP32 solve errs by
a few units of 2^-24, some 1e-7, and one with plain TF32 operands (the split
products' low parts left out) in the Schur products alone by 3.6e-6 to 5.5e-6 at
the first four shapes below, so 1e-6 tells the two apart; 2e-15 is the same
multiple of 2^-53.  One correction in FP64 then
leaves 1e-6 of the error, below the 1e-12 asked for, and a second one at most
is taken.  On real meshes an unrefined complex64 residual r contracts by r a
correction: 1e-3 is below 1e-10 after three, which leaves four for a mesh a
little worse, and never GMRES."""

from __future__ import annotations

import numpy as np
import pytest

from lithofem_b200.solver import C64, C128, DirectSolver
from tests.test_gpu_solver import CASES, system
from tests.test_gpu_sweeps import two_elements

pytestmark = pytest.mark.gpu
GATE = {C64: 1e-6, C128: 2e-15}


def solve(sv, A, vals, prec, nrhs=2):
    import torch
    v = torch.from_numpy(vals).cuda()
    assert sv.FactorDevice(v.data_ptr(), prec), sv.last_error
    rng = np.random.default_rng(len(A))
    B = rng.standard_normal((nrhs, len(A))) + 1j * rng.standard_normal((nrhs, len(A)))
    b = torch.from_numpy(B).cuda()
    x = torch.empty_like(b)
    for transpose, M in ((False, A), (True, A.T)):
        assert sv.Backsolve(nrhs, b.data_ptr(), x.data_ptr(), transpose), sv.last_error
        want = np.linalg.solve(M, B.T).T
        err = np.linalg.norm(x.cpu().numpy() - want) / np.linalg.norm(want)
        assert err <= GATE[prec], (transpose, err)


@pytest.mark.parametrize("prec", [C64, C128], ids=["c64", "c128"])
@pytest.mark.parametrize("a,s", [(33, 95), (257, 1), (513, 255), (641, 31)])
def test_unrefined_solves(a, s, prec):
    sv, A, vals = two_elements(a, s, seed=a + s, shuffled=True)
    solve(sv, A, vals, prec)
    sv.Release()


@pytest.mark.parametrize("batch_min", ["1", "1000"], ids=["batched", "per-front"])
@pytest.mark.parametrize("a,s", [(16, 16), (64, 65), (65, 64), (130, 70), (600, 49)])
def test_split_products_are_compensated(a, s, batch_min, monkeypatch):
    monkeypatch.setenv("LFSOLVE_TF32X3_MIN", "1")
    monkeypatch.setenv("LFSOLVE_BATCH_MIN", batch_min)
    sv, A, vals = two_elements(a, s, seed=5 * a + s, shuffled=True)
    solve(sv, A, vals, C64)
    sv.Release()


@pytest.mark.parametrize("split_min", [None, "1"], ids=["default", "split"])
@pytest.mark.parametrize("kcase", CASES, ids=[f"{k}-p{p}-t{t:g}" for k, p, t in CASES])
def test_corrections_of_refined_solves(kcase, split_min, monkeypatch):
    import torch
    if split_min:
        monkeypatch.setenv("LFSOLVE_TF32X3_MIN", split_min)
    monkeypatch.setenv("LFSOLVE_GMRES", "0")
    c, g, b = system(kcase)
    sv = DirectSolver(0)
    assert sv.AnalyzeAssembly(g, c.ad) and sv.FactorDevice(g._csr()[2], C64), sv.last_error
    x = torch.empty_like(b)
    for transpose in (False, True):
        ok, rel, iters = sv.SolveRefined(g, 2, b.data_ptr(), x.data_ptr(), transpose, 1e-10)
        assert ok and iters <= 4, (transpose, rel, iters)
    sv.Release()
