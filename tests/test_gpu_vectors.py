"""The element source vectors and the permittivity gradient at the edges of
their tiles: element counts that fill no block, one to three columns (pairs of
element and column are taken four a warp), each order's basis table, and rules
one point longer than the framework's and as long as a handle takes (40 points
with the curl rule's; 24 are staged at a time, eight or four a step).  A longer rule repeats points at split weights:
the same integral.

References: the oracle's right-hand side, and, as A and b are affine in the
permittivities, lambda^T (b - A u) of the oracle at eps + d less that at eps,
which the gradient's sum over d reproduces exactly.  Sums of at most 1e5 terms
of like size in 64 bits: 1e-11 of the largest entry (of the sum of moduli)."""

from __future__ import annotations

import copy
from dataclasses import replace

import numpy as np
import pytest

from lithofem_b200 import configs
from lithofem_b200.asm import AsmGpuGlobal
from oracle import oracle
from tests.test_gpu_parity import _synthetic_parts

pytestmark = pytest.mark.gpu
H = {1: 1.8, 2: 2.4, 3: 3.2}


def longer_rule(r, extra):
    """r with its first `extra` points (cyclically) given twice."""
    at = np.arange(extra) % r.nq
    times = 1 + np.bincount(at, minlength=r.nq)
    idx = np.concatenate([np.arange(r.nq), at])

    def take(a):
        return None if a is None else np.asarray(a).reshape(r.nq, -1)[idx].ravel()

    return replace(r, nq=len(idx), ip=take(r.ip), w=take(np.asarray(r.w) / times),
                   vshape=take(r.vshape), curl=take(r.curl))


def setup(p, theta, extra):
    c = configs.small_case("hole", p, theta, seed=5, h=H[p])
    ad = copy.copy(c.ad)
    if extra is None:
        extra = 40 - ad.rule_cc.nq - ad.rule_mass.nq
    ad.rule_mass = longer_rule(ad.rule_mass, extra)
    prob = copy.copy(c.prob)
    prob.elem_eps = configs.absorber_jitter(ad, prob)
    return c, ad, prob


@pytest.mark.parametrize("extra", [0, 1, None])
@pytest.mark.parametrize("p,theta", [(1, 6.0), (2, 0.0), (3, 6.0)])
def test_source_vectors(p, theta, extra):
    import torch
    c, ad, prob = setup(p, theta, extra)
    g = AsmGpuGlobal(prob)
    assert g.Init(ad, 0) and g.BuildGlobal(ad.ess)
    parts = _synthetic_parts(c, np.random.default_rng(3), 3)
    for cols, ncol in (([0, 0, 0], 1), ([1, 0, 1], 2), ([2, 0, 1], 3)):
        b = torch.full((ncol, ad.height), 7.0, dtype=torch.complex128, device="cuda")
        assert g.AssembleRHS(parts, cols, ncol, True, b.data_ptr())
        ref = oracle.rhs(ad, prob, parts, cols, ncol, ad.ess, True).reshape(ncol, -1)
        for q in range(ncol):
            err = np.abs(b[q].cpu().numpy() - ref[q]).max()
            assert err < 1e-11 * np.abs(ref[q]).max()


@pytest.mark.parametrize("extra", [0, 1, None])
@pytest.mark.parametrize("p,theta", [(1, 0.0), (2, 6.0), (3, 6.0)])
def test_permittivity_gradient(p, theta, extra):
    import torch
    c, ad, prob = setup(p, theta, extra)
    rng = np.random.default_rng(11)
    parts = _synthetic_parts(c, rng, 2)
    n = ad.height
    u, lam = (rng.standard_normal(n) + 1j * rng.standard_normal(n) for _ in range(2))
    u[ad.ess] = lam[ad.ess] = 0.0
    g = AsmGpuGlobal(prob)
    assert g.Init(ad, 0) and g.BuildGlobal(ad.ess)
    ud, ld = torch.from_numpy(u).cuda(), torch.from_numpy(lam).cuda()
    grad = torch.full((ad.ne,), 7.0, dtype=torch.complex128, device="cuda")
    assert g.EpsGradient(parts, ud.data_ptr(), ld.data_ptr(), grad.data_ptr())
    grad = grad.cpu().numpy()
    pml = np.array([prob.regions[a - 1].is_pml for a in ad.attr])
    assert np.all(grad[pml] == 0)
    I, J = oracle.csr(ad)

    def form(eps):
        q = copy.copy(prob)
        q.elem_eps = eps
        b = oracle.rhs(ad, q, parts, [0, 0], 1, ad.ess, True).reshape(-1)
        A = oracle.assemble(ad, q, I, J, ad.ess, eliminate=True)
        return lam @ b - lam @ oracle.spmv(I, J, A, u)[0]

    d = np.where(pml, 0, rng.standard_normal(ad.ne) + 1j * rng.standard_normal(ad.ne))
    diff = form(prob.elem_eps + d) - form(prob.elem_eps)
    assert abs(grad @ d - diff) < 1e-11 * np.abs(grad * d).sum() + 1e-13 * abs(form(prob.elem_eps))
