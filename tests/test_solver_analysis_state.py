"""The solver's analysis state (no GPU): an analysis that fails leaves nothing
that a later call would take for a valid one."""

from __future__ import annotations

import ctypes as ct

import numpy as np

from lithofem_b200 import configs, solver
from oracle import oracle

ERR_ARG, ERR_STATE = 1, 3


def test_a_failed_analysis_is_no_analysis():
    c = configs.small_case("slab", 1, 0.0, seed=5)
    I, J = oracle.csr(c.ad)
    s = solver.DirectSolver(0)
    L = solver.lib()
    assert s.Analyze(c.ad, I, J), s.last_error
    n = c.ad.height
    perm = np.empty(n, dtype=np.int32)
    assert L.lfsolve_get_ordering(s._s, solver._ip(perm), None) == 0
    broken = J.copy()
    broken[I[3]:I[4]] = np.arange(I[4] - I[3])        # one row's columns: not symmetric
    assert not s.Analyze(c.ad, I, broken) and s.last_error[0] == ERR_ARG
    assert L.lfsolve_get_ordering(s._s, solver._ip(perm), None) == ERR_STATE
    assert L.lfsolve_get_fronts(s._s, None, None, None, None) == ERR_STATE
    assert L.lfsolve_factor(s._s, ct.c_void_p(16), 0) == ERR_STATE
    assert s.Analyze(c.ad, I, J), s.last_error
    assert L.lfsolve_get_ordering(s._s, solver._ip(perm), None) == 0
    s.Release()


def test_a_refused_argument_keeps_the_analysis():
    """Checks that come before the ordering leave the last analysis as it is."""
    c = configs.small_case("slab", 1, 0.0, seed=5)
    I, J = oracle.csr(c.ad)
    s = solver.DirectSolver(0)
    assert s.Analyze(c.ad, I, J), s.last_error
    short = I.copy()
    short[-1] -= 1
    assert not s.Analyze(c.ad, short, J) and s.last_error[0] == ERR_ARG
    assert solver.lib().lfsolve_get_fronts(s._s, None, None, None, None) == 0
    s.Release()


def test_workspace_figure_is_what_the_factorization_takes(monkeypatch):
    """peak_front_entries: the largest even and the largest odd depth, which
    are held together but need not be neighbours (a front a group, so that the
    padded layout follows from pivots and rows: both parts to 16, fronts to 32
    entries)."""
    monkeypatch.setenv("LFSOLVE_BATCH_MIN", "1000000")
    c = configs.small_case("grating", 3, 6.0, seed=5)
    I, J = oracle.csr(c.ad)
    s = solver.DirectSolver(0)
    assert s.Analyze(c.ad, I, J), s.last_error
    f = s.Fronts()
    pad = lambda v, a: (v.astype(np.int64) + a - 1) // a * a
    entries = pad((pad(f["k"], 16) + pad(f["m"] - f["k"], 16)) ** 2, 32)
    depth = np.bincount(f["depth"], weights=entries).astype(np.int64)
    held = depth[::2].max() + depth[1::2].max()
    assert held > (depth[1:] + depth[:-1]).max()      # not neighbours here
    assert s.Stats()["peak_front_entries"] == held
    s.Release()
