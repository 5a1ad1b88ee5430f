"""What a program that uses this framework has it do, as measurable cases.

A user meshes a periodic lithography cell, assembles its Maxwell system for
one set of material values after another, factors it, solves for the sources
and the adjoint, and reads the orders and the gradient.  The cases are the
calls of that loop through the public entry points (``lithofem_b200.asm``,
``lithofem_b200.solver``, ``lithofem_b200.adjoint``), from the smallest
meshes, where latency counts, to the 1.35M-DOF line grating of
``configs.config(3)``.  What the seed changes is what changes from one
iteration to the next: the absorber elements' permittivity and the vectors.

``exact`` restates each result in 64-bit torch, from the mesh arrays and the
element's reference tables alone.
"""

from __future__ import annotations

import copy
import math
from functools import lru_cache

import numpy as np
import torch

from lithofem_b200 import configs, incident, ndbasis
from lithofem_b200.adjoint import EffAdjoint
from lithofem_b200.asm import AsmBatch, AsmGpuGlobal
from lithofem_b200.solver import C64, C128, DirectSolver

DEV = "cuda:0"
CPLX = torch.complex128
STACKS = {"slab": configs.slab_stack, "hole": configs.contact_hole_stack,
          "grating": configs.line_grating_stack}
ITERATIONS = ("assemble", "fresh", "ends", "orders", "factor", "resolve", "adjoint")


def listed():
    return [
        # a convergence study's coarse mesh: launches and host time are all there is
        dict(name="assemble_p1_slab_small", kind="assemble", geom="slab", p=1, theta=0.0, ndof=3e3),
        # the contact hole with per-element permittivity, the next design on a kept handle
        dict(name="assemble_p2_hole", kind="assemble", geom="hole", p=2, theta=6.0, ndof=300e3),
        # the largest mesh: the 1.35M-DOF line grating
        dict(name="assemble_p3_grating", kind="assemble", geom="grating", p=3, theta=6.0, ndof=1.3e6),
        # many uneven meshes of mixed order at once
        dict(name="batch_polygons", kind="batch", count=16, scale=0.25, theta=6.0, mesh=0),
        # a design iteration that makes a new handle from host arrays: upload, device CSR
        # structure, values and right-hand side
        dict(name="fresh_p2_hole", kind="fresh", geom="hole", p=2, theta=6.0, ndof=300e3),
        # the two ends of an iteration: s and p sources in, the permittivity gradient out
        dict(name="ends_p3_grating", kind="ends", geom="grating", p=3, theta=6.0, ndof=300e3),
        # post-processing: reflection and transmission planes and their orders
        dict(name="orders_p2_hole", kind="orders", geom="hole", p=2, theta=6.0, ndof=110e3, nx=48,
             ny=48),
        # new values on a known structure: factor, then s and p fields (the default, mixed precision)
        dict(name="factor_c64_p1_slab_small", kind="factor", geom="slab", p=1, theta=6.0, ndof=6e3,
             prec="c64"),
        dict(name="factor_c64_p3_grating", kind="factor", geom="grating", p=3, theta=6.0, ndof=500e3,
             prec="c64"),
        # the same in plain FP64, factors used as they are
        dict(name="factor_c128_p2_hole", kind="factor", geom="hole", p=2, theta=6.0, ndof=120e3,
             prec="c128"),
        # further sources and an adjoint on kept factors
        dict(name="resolve_p3_grating", kind="resolve", geom="grating", p=3, theta=6.0, ndof=300e3),
        # one whole inverse-design step: value and gradient of an order's efficiency
        dict(name="adjoint_p2_hole", kind="adjoint", geom="hole", p=2, theta=6.0, ndof=60e3),
    ]


# kind: range of the DOF target, up to what the listed ones reach in time
RANGES = {"assemble": (1.5e3, 900e3), "fresh": (3e3, 300e3), "ends": (3e3, 300e3),
          "orders": (5e3, 200e3), "factor": (3e3, 300e3), "resolve": (3e3, 300e3),
          "adjoint": (3e3, 60e3)}


def draw(rng):
    kind = rng.choice(ITERATIONS + ("batch",))
    theta = rng.choice([0.0, round(rng.uniform(1.0, 25.0), 2)])
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(3, 16), scale=round(rng.uniform(0.05, 0.25), 4),
                    theta=theta, mesh=rng.randint(1, 10 ** 6))
    lo, hi = RANGES[kind]
    case = dict(kind=kind, geom=rng.choice(sorted(STACKS)), p=rng.randint(1, 3), theta=theta,
                ndof=round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if kind == "orders":
        case.update(nx=rng.randint(9, 64), ny=rng.randint(9, 64))
    if kind == "factor":
        case["prec"] = rng.choice(["c64", "c128"])
        if case["prec"] == "c128":
            case["ndof"] = min(case["ndof"], 150e3)
    if kind in ("assemble", "fresh") and case["p"] == 1:
        case["ndof"] = min(case["ndof"], 200e3)      # p = 1 meshes: many elements a DOF
    if kind == "adjoint" and case["geom"] == "slab":
        case["geom"] = "hole"
    return case


# -- what the program has in hand -------------------------------------------

@lru_cache(maxsize=3)
def _mesh(geom, p, theta, ndof):
    return configs.make_case(geom, STACKS[geom](), p, theta, ndof)


@lru_cache(maxsize=2)
def _batch_meshes(count, scale, theta, mesh):
    return configs.batch_config(scale=scale, n=count, seed=configs.SEED + mesh, theta=theta)


def _meshes(case):
    if case["kind"] == "batch":
        return _batch_meshes(case["count"], case["scale"], case["theta"], case["mesh"])
    return [_mesh(case["geom"], case["p"], case["theta"], case["ndof"])]


def _problem(c, seed):
    """The mesh's problem with this iteration's absorber permittivities."""
    prob = copy.copy(c.prob)
    prob.elem_eps = configs.absorber_jitter(c.ad, c.prob, seed=seed)
    return prob


def _parts(c, pols):
    return [incident.planewave_parts(c.stack, c.theta, 0.0, q) for q in pols]


def _vector(n, seed):
    rng = np.random.default_rng(seed)
    return torch.from_numpy(rng.standard_normal(n) + 1j * rng.standard_normal(n)).to(DEV)


def _handle(c, prob):
    g = AsmGpuGlobal(prob)
    assert g.Init(c.ad, 0) and g.BuildGlobal(c.ad.ess)
    return g


class _Borrowed:
    """A handle's device array that keeps the handle alive."""

    def __init__(self, view, owner):
        self.__cuda_array_interface__, self.owner = view.__cuda_array_interface__, owner


def _csr(g):
    return [torch.as_tensor(_Borrowed(v, g), device=DEV) for v in g.DeviceCsrViews()]


def _planes(c):
    """Reflection and transmission plane, in the top and the bottom half wavelength."""
    st, parts = c.stack, _parts(c, "s")
    top, bot = parts[0][-1], parts[0][0]
    bg_top = top.B * np.exp(1j * top.qB * (st.z_max - top.zB))
    bg_bot = (bot.A * np.exp(1j * bot.qA * (st.z_min - bot.zA))
              + bot.B * np.exp(1j * bot.qB * (st.z_min - bot.zB)))
    return [dict(z=st.z_max - 4.7, z_ref=st.z_max, eps=1.0, direction=1, bg00=bg_top),
            dict(z=st.z_min + 4.3, z_ref=st.z_min, eps=st.eps_bg_of_slab(0), direction=-1,
                 bg00=bg_bot)]


def _order_args(c):
    pr = c.prob
    qz = math.sqrt(pr.k0 ** 2 - pr.kx ** 2 - pr.ky ** 2)
    return dict(lx=c.stack.lx, ly=c.stack.ly, k0=pr.k0, kx=pr.kx, ky=pr.ky,
                inc_flux=0.5 * qz / pr.k0 * c.stack.lx * c.stack.ly)


def _z_objective(c):
    st = c.stack
    return st.z_max - 0.25 * (st.z_max - st.slabs[-2])


def prepare(case, seed):
    kind = case["kind"]
    cs = _meshes(case)
    c = cs[0]
    n = c.ad.height
    s = dict(kind=kind, case=c)
    if kind == "batch":
        s["g"] = [_handle(m, _problem(m, seed + i)) for i, m in enumerate(cs)]
        s["batch"] = AsmBatch(s["g"])
        s["vals"] = [_csr(g)[2] for g in s["g"]]
        return s
    prob = s["prob"] = _problem(c, seed)
    if kind == "adjoint":
        s["eps"] = prob.elem_eps
        s["adj"] = EffAdjoint(c.ad, c.prob, _parts(c, "s"), _z_objective(c), c.stack.lx,
                              c.stack.ly, 16, 16)
        return s
    if kind == "fresh":
        s["parts"] = _parts(c, "s")
        s["b"] = torch.empty(n, dtype=CPLX, device=DEV)
        return s
    g = s["g"] = _handle(c, prob)
    if kind == "assemble":
        s["vals"] = _csr(g)[2]
    elif kind == "ends":
        s["parts"] = _parts(c, "sp")
        s["b"] = torch.empty(2, n, dtype=CPLX, device=DEV)
        s["u"], s["lam"] = _vector(n, seed), _vector(n, seed + 1)
        s["grad"] = torch.empty(c.ad.ne, dtype=CPLX, device=DEV)
    elif kind == "orders":
        nx, ny = s["nx"], s["ny"] = case["nx"], case["ny"]
        assert g.SetBasis(ndbasis.nd_element(c.p))
        s["planes"], s["args"] = _planes(c), _order_args(c)
        s["u"] = _vector(n, seed)
        s["E"] = torch.empty(2, ny, nx, 3, dtype=CPLX, device=DEV)
        s["H"] = torch.empty_like(s["E"])
        s["coef"] = torch.empty_like(s["E"])
        s["eff"] = torch.empty(2, ny, nx, dtype=torch.float64, device=DEV)
    else:                                     # factor, resolve
        assert g.Assemble(True)
        s["b"] = torch.empty(2, n, dtype=CPLX, device=DEV)
        assert g.AssembleRHS(_parts(c, "sp"), [0, 1], 2, True, s["b"].data_ptr())
        s["x"] = torch.empty_like(s["b"])
        s["vals"] = g.DeviceCsrViews()[2].__cuda_array_interface__["data"][0]
        s["lu"] = DirectSolver(0)
        assert s["lu"].AnalyzeAssembly(g, c.ad)
        s["prec"] = C128 if case.get("prec") == "c128" else C64
        if kind == "resolve":
            assert g.SetBasis(ndbasis.nd_element(c.p))
            s["c"] = torch.empty(n, dtype=CPLX, device=DEV)
            assert g.PlaneSeed(c.stack.lx, c.stack.ly, _z_objective(c), 16, 16, seed % 2, 0, 0,
                               s["c"].data_ptr())
            s["lam"] = torch.empty_like(s["c"])
            assert s["lu"].FactorDevice(s["vals"], C64)
    return s


# -- one pass ------------------------------------------------------------------

def run(s):
    kind, c = s["kind"], s["case"]
    if kind == "batch":
        assert s["batch"].Assemble(True)
        return {"vals": s["vals"]}
    if kind == "adjoint":
        eta, g_re, g_im = s["adj"].value_and_grad(s["eps"])
        return {"eta": eta, "g_re": g_re, "g_im": g_im}
    if kind == "fresh":
        g = s["g"] = AsmGpuGlobal(s["prob"])
        assert g.Init(c.ad, 0) and g.BuildGlobal(c.ad.ess) and g.Assemble(True)
        assert g.AssembleRHS(s["parts"], [0], 1, True, s["b"].data_ptr())
        rowptr, cols, vals = _csr(g)
        return {"rowptr": rowptr, "cols": cols, "vals": vals, "b": s["b"]}
    g = s["g"]
    if kind == "assemble":
        assert g.Assemble(True)
        return {"vals": s["vals"]}
    if kind == "ends":
        assert g.AssembleRHS(s["parts"], [0, 1], 2, True, s["b"].data_ptr())
        assert g.EpsGradient(s["parts"][:1], s["u"].data_ptr(), s["lam"].data_ptr(),
                             s["grad"].data_ptr())
        return {"b": s["b"], "grad": s["grad"]}
    if kind == "orders":
        st, nx, ny = c.stack, s["nx"], s["ny"]
        assert g.SamplePlanes(st.lx, st.ly, [q["z"] for q in s["planes"]], nx, ny,
                              s["u"].data_ptr(), s["E"].data_ptr(), s["H"].data_ptr())
        assert g.PlaneOrders(nx, ny, s["E"].data_ptr(), s["planes"], s["args"],
                             s["coef"].data_ptr(), s["eff"].data_ptr())
        return {"E": s["E"], "H": s["H"], "coef": s["coef"], "eff": s["eff"]}
    lu, b, x = s["lu"], s["b"], s["x"]
    if kind == "factor":
        assert lu.FactorDevice(s["vals"], s["prec"]), lu.last_error
        if s["prec"] == C128:
            assert lu.Backsolve(2, b.data_ptr(), x.data_ptr()), lu.last_error
        else:
            assert lu.SolveRefined(g, 2, b.data_ptr(), x.data_ptr())[0], lu.last_error
        return {"x": x}
    assert lu.SolveRefined(g, 2, b.data_ptr(), x.data_ptr())[0], lu.last_error
    assert lu.SolveRefined(g, 1, s["c"].data_ptr(), s["lam"].data_ptr(), True)[0], lu.last_error
    return {"x": x, "lam": s["lam"]}


# -- what a pass cannot do without ---------------------------------------------

def _nnz(ad):
    """Couplings an H(curl) row has on these meshes: distinct entries of the element matrices."""
    return {1: 16.2, 2: 43.2, 3: 85.5}[ad.p] * ad.height


def work(case):
    kind = case["kind"]
    nbytes = flops = 0.0
    for c in _meshes(case):
        ad = c.ad
        n, ne, nd, nnz = ad.height, ad.ne, ad.nd, _nnz(ad)
        geometry = ne * (9 + 9 + 1 + 3) * 8.0 + ne * nd * 4.5 + ne * 16
        element = 4.0 * nd * nd * 30 * ne           # 30 coefficient terms an entry
        if kind in ("assemble", "batch", "fresh"):
            nbytes += geometry + 16 * nnz
            flops += element
        if kind == "fresh":
            nbytes += 4 * nnz + 16 * n
        if kind == "ends":
            nbytes += geometry + 16 * (2 * n + 2 * n + ne)
            flops += ne * ad.rule_mass.nq * nd * 3 * 16.0
        if kind == "orders":
            pts = 2.0 * case["nx"] * case["ny"]
            nbytes += geometry / nd + pts * 16 * (nd + 9) + pts * 8
            flops += pts * nd * 48 + pts * 3 * 8 * (case["nx"] + case["ny"])
        if kind in ("factor", "resolve", "adjoint"):
            # nested dissection of a cell of this shape: 30 n^(4/3) entries, 70 n^2 operations
            es = 16 if case.get("prec") == "c128" else 8
            entries = 30.0 * n ** (4 / 3)
            sweeps = 1 if es == 16 else {"factor": 3, "resolve": 6, "adjoint": 6}[kind]
            nbytes += 16 * nnz + sweeps * (entries * es) + 64 * n
            flops += sweeps * entries * 8
            if kind != "resolve":
                flops += 70.0 * n * n
                nbytes += entries * es
    return {"bytes": nbytes, "flops": flops}


# -- the same results in plain 64-bit torch ------------------------------------

def _t(a, shape=None):
    t = torch.from_numpy(np.ascontiguousarray(a)).to(DEV)
    return t if shape is None else t.reshape(shape)


class _Exact:
    """The system's forms on the mesh arrays, elements in chunks."""

    def __init__(self, ad, prob):
        self.ad, self.prob, self.nd, self.ne = ad, prob, ad.nd, ad.ne
        self.J, self.Ji = _t(ad.J, (-1, 3, 3)), _t(ad.Jinv, (-1, 3, 3))
        self.det, self.v0 = _t(ad.detJ), _t(ad.v0, (-1, 3))
        self.dof = _t(ad.dof, (-1, ad.nd)).long()
        self.sign = _t(ad.sign, (-1, ad.nd))
        self.eps = _t(np.asarray(prob.elem_eps, dtype=complex))
        self.ess = _t(ad.ess).long()
        n_bot = n_top = 1.0
        for r in prob.regions:
            if r.is_pml:
                n = abs(np.sqrt(complex(r.eps)))
                n_bot, n_top = (n_bot, n) if r.pml_top else (n, n_top)
        f = -math.log(prob.pml_target) * (prob.pml_order + 1) / (2 * prob.k0 * prob.pml_thick)
        self.smax = f / n_bot, f / n_top

    def chunks(self):
        size = min(30_000, 3_000_000 // (self.nd * self.nd))
        return [slice(a, min(self.ne, a + size)) for a in range(0, self.ne, size)]

    def heights(self, el, rule):
        ip = _t(rule.ip, (-1, 3))
        return self.v0[el, 2:3] + torch.einsum("ej,qj->eq", self.J[el, 2], ip)

    def stretch(self, z):
        p = self.prob
        d = torch.where(z < p.z_min, (p.z_min - z) / p.pml_thick, (z - p.z_max) / p.pml_thick)
        smax = torch.where(z < p.z_min, torch.full_like(z, self.smax[0]), self.smax[1])
        s = smax * d.clamp(0.0, 1.0) ** p.pml_order
        return torch.complex(torch.ones_like(z), torch.where(d > 0, s, torch.zeros_like(s)))

    def values(self, el, rule):        # (e, q, k, 3) physical basis values, curls
        v = _t(rule.vshape, (rule.nq, self.nd, 3))
        return torch.einsum("qkj,eji->eqki", v, self.Ji[el])

    def curls(self, el, rule):
        v = _t(rule.curl, (rule.nq, self.nd, 3))
        return torch.einsum("qkj,eij->eqki", v, self.J[el]) / self.det[el, None, None, None]

    def to_dofs(self, el):
        """(e, k, l): the element's functions in terms of the global ones (signs, face pairs)."""
        ad, p = self.ad, self.ad.p
        e = torch.arange(self.ne, device=DEV)[el]
        T = torch.eye(self.nd, dtype=torch.float64, device=DEV).repeat(len(e), 1, 1)
        if p > 1:
            G = np.array([[0.0, 0.0], [1.0, 0.0], [0.0, 1.0]])
            perms = ((0, 1, 2), (1, 0, 2), (1, 2, 0), (2, 1, 0), (2, 0, 1), (0, 2, 1))
            M = np.array([np.array([G[b] - G[a], G[c] - G[a]]).T for a, b, c in perms])
            fo = _t(ad.fo, (-1, 4))[el].long()
            for f in range(4):
                blk = _t(M)[fo[:, f]]
                for i in range(p * (p - 1) // 2):
                    d = 6 * p + f * p * (p - 1) + 2 * i
                    T[:, d:d + 2, d:d + 2] = blk
        return T * self.sign[el][:, :, None]

    def coefficients(self, el, rule):
        s = self.stretch(self.heights(el, rule))
        w = _t(rule.w)[None, :] * self.det[el][:, None]
        return w, torch.stack([s, s, 1 / s], -1), torch.stack([1 / s, 1 / s, s], -1)

    def matrix(self):
        """(rowptr, cols, vals) of the eliminated system."""
        ad, pr = self.ad, self.prob
        n = ad.height
        K = _t(np.array([[0, 0, pr.ky], [0, 0, -pr.kx], [-pr.ky, pr.kx, 0]])).to(CPLX)
        pat = torch.cat([torch.unique((self.dof[el, :, None] * n + self.dof[el, None, :]).reshape(-1))
                         for el in self.chunks()])
        pat = torch.unique(pat)
        vals = torch.zeros(len(pat), 2, dtype=torch.float64, device=DEV)
        for el in self.chunks():
            X = self.curls(el, ad.rule_cc).to(CPLX)
            w, _, li = self.coefficients(el, ad.rule_cc)
            A = self.contract(X, X * (w[..., None] * li)[:, :, None, :])
            V, X = (f(el, ad.rule_mass).to(CPLX) for f in (self.values, self.curls))
            w, lam, li = self.coefficients(el, ad.rule_mass)
            D = torch.diag_embed(-pr.k0 ** 2 * self.eps[el][:, None, None] * lam)
            D = D - torch.einsum("rt,eqt,tc->eqrc", K, li, K)
            A = A + self.contract(V, torch.einsum("eqrc,eqkc->eqkr", w[..., None, None] * D, V))
            D = 1j * w[..., None, None] * K * li[:, :, None, :]
            A = A + self.contract(V, torch.einsum("eqrc,eqkc->eqkr", D, X))
            D = 1j * w[..., None, None] * li[..., None] * K
            A = A + self.contract(X, torch.einsum("eqrc,eqkc->eqkr", D, V))
            T = self.to_dofs(el).to(CPLX)
            A = T @ A @ T.transpose(1, 2)
            at = torch.searchsorted(pat, (self.dof[el, :, None] * n
                                          + self.dof[el, None, :]).reshape(-1))
            vals.index_add_(0, at, torch.view_as_real(A.reshape(-1)))
        row, col = pat // n, pat % n
        is_ess = torch.zeros(n, dtype=torch.bool, device=DEV)
        is_ess[self.ess] = True
        gone = is_ess[row] | is_ess[col]
        vals[gone] = 0.0
        vals[gone & (row == col), 0] = 1.0
        rowptr = torch.searchsorted(row, torch.arange(n + 1, device=DEV))
        return rowptr, col, torch.view_as_complex(vals)

    @staticmethod
    def contract(X, Y):
        e, q, k, _ = X.shape
        flat = lambda a: a.permute(0, 2, 1, 3).reshape(e, k, 3 * q)  # noqa: E731
        return flat(X) @ flat(Y).transpose(1, 2)

    def wave(self, part, slab, z):
        """(e, q, 3) incident envelope of one part in the elements' slabs."""
        out = 0
        for q0, z0, amp in (("qA", "zA", "A"), ("qB", "zB", "B")):
            q, zz, a = (_t(np.array([getattr(w, f) for w in part]))[slab] for f in (q0, z0, amp))
            out = out + torch.exp(1j * q[:, None] * (z - zz[:, None]))[..., None] * a[:, None, :]
        return out

    def background(self):
        """Per element: slab, eps of its slab's background, and whether it lies in the PML."""
        pr = self.prob
        bg = {r.slab: complex(r.eps) for r in pr.regions if r.kind == 0}
        attr = self.ad.attr - 1
        slab = np.array([r.slab for r in pr.regions])[attr]
        pml = np.array([r.is_pml for r in pr.regions])[attr]
        known = ~pml & np.isin(slab, list(bg))
        eps = np.array([bg.get(i, 0j) for i in slab])
        return _t(slab).long(), _t(eps), _t(pml), _t(known)

    def rhs(self, parts, columns):
        ad, rule = self.ad, self.ad.rule_mass
        slab, bg, _, known = self.background()
        delta = torch.where(known, self.eps - bg, 0.0)
        b = torch.zeros(columns, ad.height, 2, dtype=torch.float64, device=DEV)
        for el in self.chunks():
            z = self.heights(el, rule)
            w = _t(rule.w)[None, :] * self.det[el][:, None]
            V, T = self.values(el, rule).to(CPLX), self.to_dofs(el).to(CPLX)
            for c in range(columns):
                E = self.wave(parts[c], slab[el], z)
                E = E * (self.prob.k0 ** 2 * delta[el])[:, None, None] * w[..., None]
                be = torch.einsum("ekl,el->ek", T, torch.einsum("eqki,eqi->ek", V, E))
                b[c].index_add_(0, self.dof[el].reshape(-1), torch.view_as_real(be.reshape(-1)))
        b[:, self.ess] = 0.0
        return torch.view_as_complex(b)

    def gradient(self, parts, u, lam):
        rule, k2 = self.ad.rule_mass, self.prob.k0 ** 2
        slab, _, pml, known = self.background()
        out = torch.zeros(self.ne, dtype=CPLX, device=DEV)
        for el in self.chunks():
            V, T = self.values(el, rule).to(CPLX), self.to_dofs(el).to(CPLX)
            w, L, _ = self.coefficients(el, rule)
            U, Z = (torch.einsum("eqki,ek->eqi", V, torch.einsum("elk,el->ek", T, f[self.dof[el]]))
                    for f in (u, lam))
            src = sum(self.wave(p, slab[el], self.heights(el, rule)) for p in parts)
            src = src * known[el][:, None, None]
            out[el] = k2 * torch.einsum("eq,eqi,eqi->e", w.to(CPLX), Z, L * U + src)
        return torch.where(pml, 0.0, out)

    def sample(self, el, xi, u):
        """E and curl E of u at reference points xi of the elements el."""
        b = ndbasis.nd_element(self.ad.p)
        m = torch.stack([(xi ** _t(np.array(e))).prod(-1) for e in b.monos], -1)
        v = torch.einsum("pm,kdm->pkd", m, _t(b.coef))
        w = torch.einsum("pm,kdm->pkd", m, _t(b._curl_coef))
        loc = torch.einsum("plk,pl->pk", self.to_dofs(el).to(CPLX), u[self.dof[el]])
        E = torch.einsum("pk,pkj,pji->pi", loc, v.to(CPLX), self.Ji[el].to(CPLX))
        H = torch.einsum("pk,pkj,pij->pi", loc, w.to(CPLX), self.J[el].to(CPLX))
        return E, H / self.det[el, None]

    def locate(self, X):
        el, ref = [], []
        for x in X.split(32):
            d = x[:, None, :] - self.v0[None]
            xi = torch.einsum("eij,pej->pei", self.Ji, d)
            inside = torch.minimum(xi.min(-1).values, 1 - xi.sum(-1))
            best = inside.argmax(1)
            el.append(best)
            ref.append(xi[torch.arange(len(x), device=DEV), best])
        return torch.cat(el), torch.cat(ref)


def _exact_orders(case, c, ex, u):
    nx, ny, st, a = case["nx"], case["ny"], c.stack, _order_args(c)
    planes = _planes(c)
    x = (torch.arange(nx, device=DEV, dtype=torch.float64) + 0.5) * st.lx / nx + 3.1e-7
    y = (torch.arange(ny, device=DEV, dtype=torch.float64) + 0.5) * st.ly / ny + 1.7e-7
    out = {"E": [], "H": [], "coef": [], "eff": []}
    for q in planes:
        X = torch.stack([x.repeat(ny), y.repeat_interleave(nx), torch.full_like(x, q["z"] - 4.9e-7
                                                                                ).repeat(ny)], -1)
        E, H = ex.sample(*ex.locate(X), u)
        E, H = E.reshape(ny, nx, 3), H.reshape(ny, nx, 3)
        coef = torch.fft.fft2(E, dim=(0, 1)) / (nx * ny)
        half = lambda n: _t(np.array([i if i <= n // 2 else i - n for i in range(n)],  # noqa: E731
                                     dtype=float))
        kx = (a["kx"] + 2 * math.pi / st.lx * half(nx))[None, :].expand(ny, nx)
        ky = (a["ky"] + 2 * math.pi / st.ly * half(ny))[:, None].expand(ny, nx)
        qz = torch.sqrt(a["k0"] ** 2 * complex(q["eps"]) - kx ** 2 - ky ** 2 + 0j)
        qz = torch.where(qz.imag < 0, -qz, qz)
        cc = coef * torch.exp(-1j * q["direction"] * qz * (q["z"] - q["z_ref"]))[..., None]
        cc[0, 0] += _t(np.asarray(q["bg00"], dtype=complex))
        k = torch.stack([kx + 0j, ky + 0j, q["direction"] * qz], -1)
        h = torch.linalg.cross(k, cc) / a["k0"]
        flux = 0.5 * torch.linalg.cross(cc, h.conj())[..., 2].real * st.lx * st.ly
        for name, v in zip(("E", "H", "coef", "eff"),
                           (E, H, coef, q["direction"] * flux / a["inc_flux"])):
            out[name].append(v)
    return {name: torch.stack(v) for name, v in out.items()}


DENSE = 14_000      # rows up to which the system is solved densely


def exact(case, seed):
    kind = case["kind"]
    cs = _meshes(case)
    if kind == "batch":
        return {"vals": [_Exact(m.ad, _problem(m, seed + i)).matrix()[2]
                         for i, m in enumerate(cs)]}
    c = cs[0]
    n = c.ad.height
    ex = _Exact(c.ad, _problem(c, seed))
    if kind == "assemble":
        return {"vals": ex.matrix()[2]}
    if kind == "fresh":
        return {"rowptr": None, "cols": None, "vals": ex.matrix()[2], "b": ex.rhs(_parts(c, "s"), 1)[0]}
    if kind == "ends":
        parts = _parts(c, "sp")
        return {"b": ex.rhs(parts, 2),
                "grad": ex.gradient(parts[:1], _vector(n, seed), _vector(n, seed + 1))}
    if kind == "orders":
        return _exact_orders(case, c, ex, _vector(n, seed))
    if kind != "factor" or n > DENSE:
        return None                            # a factorization of its own, at the size of this one
    rowptr, col, vals = ex.matrix()
    A = torch.zeros(n, n, dtype=CPLX, device=DEV)
    A[torch.repeat_interleave(torch.arange(n, device=DEV), rowptr.diff()), col] = vals
    x = torch.linalg.solve(A, ex.rhs(_parts(c, "sp"), 2).T)
    return {"x": x.T.contiguous()}
