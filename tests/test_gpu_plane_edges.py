"""Plane location, sampling and orders at the edges of their blocks: 16 points
a block against 256 candidate elements at a time, 4, 16 or 32 lanes a point
(p = 1, 2, 3), sums shared by eight lanes.

Samples: at single points against the basis evaluated on the host in the
element that holds the point (64-bit sums of at most 45 terms of like size:
1e-12 of the largest).  Orders: against numpy's FFT (sums of nx ny terms in
another order: 1e-13 of the largest)."""

from __future__ import annotations

import numpy as np
import pytest

from lithofem_b200 import configs, ndbasis, space
from lithofem_b200.asm import AsmGpuGlobal

pytestmark = pytest.mark.gpu


def host_sample(ad, u, pts):
    """E at pts (element with the largest smallest barycentric coordinate)."""
    Ji, v0 = ad.Jinv.reshape(-1, 3, 3), ad.v0.reshape(-1, 3)
    dof, sg = ad.dof.reshape(ad.ne, -1), ad.sign.reshape(ad.ne, -1)
    el, p = ndbasis.nd_element(ad.p), ad.p
    out = []
    for x in pts:
        xi = np.einsum("eij,ej->ei", Ji, x - v0)
        e = int(np.argmax(np.minimum(1 - xi.sum(1), xi.min(1))))
        loc = sg[e] * u[dof[e]]
        if p > 1:
            fo = ad.fo.reshape(ad.ne, 4)[e]
            for f in range(4):
                M = space.face_tinv(fo[f])
                for i in range(p * (p - 1) // 2):
                    d0 = 6 * p + f * p * (p - 1) + 2 * i
                    loc[d0:d0 + 2] = M @ loc[d0:d0 + 2]
        out.append(loc @ (el.vshape(xi[e][None])[0] @ Ji[e]))
    return np.array(out)


@pytest.mark.parametrize("nx,ny", [(1, 1), (5, 3), (17, 2), (16, 9)])
@pytest.mark.parametrize("p", [1, 2, 3])
def test_samples(p, nx, ny):
    import torch
    c = configs.small_case("hole", p, 6.0, seed=3, h={1: 1.8, 2: 2.4, 3: 3.2}[p])
    g = AsmGpuGlobal(c.prob)
    assert g.Init(c.ad, 0) and g.BuildGlobal(c.ad.ess) and g.SetBasis(ndbasis.nd_element(p))
    rng = np.random.default_rng(p)
    u = rng.standard_normal(c.ad.height) + 1j * rng.standard_normal(c.ad.height)
    ud = torch.from_numpy(u).cuda()
    st, zs = c.stack, [1.3, 7.9, 10.4]
    E = torch.zeros(len(zs), ny, nx, 3, dtype=torch.complex128, device="cuda")
    assert g.SamplePlanes(st.lx, st.ly, zs, nx, ny, ud.data_ptr(), E.data_ptr())
    # the sampler's fixed nudges keep points off element faces
    pts = [((i + 0.5) * st.lx / nx + 3.1e-7, (j + 0.5) * st.ly / ny + 1.7e-7, z - 4.9e-7)
           for z in zs for j in range(ny) for i in range(nx)]
    ref = host_sample(c.ad, u, np.array(pts)).reshape(E.shape)
    assert np.abs(E.cpu().numpy() - ref).max() < 1e-12 * np.abs(ref).max()
    g.Release()


@pytest.mark.parametrize("nx,ny,nz", [(1, 1, 1), (1, 17, 2), (33, 1, 3), (7, 9, 1), (64, 48, 2),
                                      (2, 130, 1)])
def test_orders(nx, ny, nz):
    import torch
    c = configs.small_case("slab", 1, 0.0)
    g = AsmGpuGlobal(c.prob)
    assert g.Init(c.ad, 0) and g.BuildGlobal(c.ad.ess)
    rng = np.random.default_rng(nx)
    E = rng.standard_normal((nz, ny, nx, 3)) + 1j * rng.standard_normal((nz, ny, nx, 3))
    Ed = torch.from_numpy(E).cuda()
    coef = torch.zeros(nz, ny, nx, 3, dtype=torch.complex128, device="cuda")
    eff = torch.zeros(nz, ny, nx, dtype=torch.float64, device="cuda")
    planes = [dict(z=1.0 + i, z_ref=2.0, eps=1.0 + 0.2j * i, direction=1 - 2 * (i % 2))
              for i in range(nz)]
    args = dict(lx=20.0, ly=14.0, k0=0.46, kx=0.03, ky=0.02, inc_flux=1.0)
    assert g.PlaneOrders(nx, ny, Ed.data_ptr(), planes, args, coef.data_ptr(), eff.data_ptr())
    ref = np.fft.fft2(E, axes=(1, 2)) / (nx * ny)
    assert np.abs(coef.cpu().numpy() - ref).max() < 1e-13 * np.abs(ref).max()
    assert torch.isfinite(eff).all()
    g.Release()
