"""Workloads of the element path: the calls a finite-element program makes on
libfem_gpu, over the range of sizes, spline orders and cell shapes it has.

Kinds of case (every case is a dict with "kind"):
  plane    2-D plane strain on a uniform QUAD4 mesh, clamp and traction:
           Jacobian and residual into the CSR (one Newton step of a plate)
  solid    3-D elasticity on an HEX8 mesh, rectangular or distorted cells, E per
           element: Jacobian and residual, or the residual alone (line search)
  simp     3-D density problem (E = rho^3 at the Gauss points), clamp and
           traction: one assembly of a topology-optimisation iteration
  apply    matrix-free Jacobian-vector product of the 3-D solid
  xfem     two-phase level-set model: uncut cells, cut clusters, interface and
           ghost penalty in one batched call
  adjoint  shape sensitivities of the level-set model: dR/dp contracted with
           the adjoint and the chain to the B-spline coefficients
  mgsolve  density problem solved with flexible CG and the multigrid V-cycle,
           hierarchy included (the operator changes in every design iteration)
  pcg      plane-strain system solved with Jacobi-PCG

Element data (E, densities, displacements) are drawn from the seed; a level
set is the case's own, since it decides the output sizes.  `exact` restates the
weak forms in plain torch, FP64.
"""
import math

import numpy as np
import torch

import moris_gb300 as mg
from moris_gb300 import learned, multigrid, sensitivity, workloads, xtk

F64 = torch.float64
NU = 0.3


# --------------------------------------------------------------------------
# cases
def listed():
    return [
        # a plate a user checks a script with: launch and synchronisation latency
        dict(name="plane_small", kind="plane", nx=24, ny=17, order=1),
        # an ordinary 2-D model with smooth extraction
        dict(name="plane_quadratic", kind="plane", nx=257, ny=130, order=2),
        # a small solid with odd, unequal edges
        dict(name="solid_small", kind="solid", nx=15, ny=13, nz=11, order=2, rect=True, jacobian=True),
        # the benchmark's size: 306 M nonzeros
        dict(name="solid_large", kind="solid", nx=64, ny=64, nz=64, order=2, rect=True, jacobian=True),
        # body-fitted cells (no constant Jacobian)
        dict(name="solid_distorted", kind="solid", nx=26, ny=23, nz=21, order=2, rect=False, jacobian=True),
        # assembly of a density problem in an optimisation loop
        dict(name="simp_assembly", kind="simp", n=96),
        # matrix-free Krylov products
        dict(name="apply_quadratic", kind="apply", nx=48, ny=47, nz=45, order=2, rect=True),
        # level-set model, linear splines (every design iteration assembles it)
        dict(name="xfem_linear", kind="xfem", n=64, order=1, spheres=40, geometry=3),
        # level-set model, quadratic splines
        dict(name="xfem_quadratic", kind="xfem", n=22, order=2, spheres=12, geometry=5),
        # sensitivities of the level-set model
        dict(name="adjoint", kind="adjoint", n=44, ncoef=24, order=1, geometry=7),
        # linear solve of the density problem
        dict(name="multigrid_solve", kind="mgsolve", n=64),
        # small solve: four launches an iteration
        dict(name="pcg_small", kind="pcg", nx=64, ny=64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plane", "plane", "solid", "solid", "solid", "simp", "apply", "xfem", "xfem", "adjoint",
                       "mgsolve", "pcg"])
    if kind == "plane":
        return dict(kind=kind, nx=_log(rng, 6, 300), ny=_log(rng, 6, 300), order=rng.choice([1, 2, 3]))
    if kind == "solid":
        rect = rng.random() < 0.7
        m = 62 if rect else 26
        order = rng.choice([1, 2, 2])
        return dict(kind=kind, nx=_log(rng, 5, m), ny=_log(rng, 5, m), nz=_log(rng, 5, m), order=order, rect=rect,
                    jacobian=rng.random() < 0.75)
    if kind == "simp":
        return dict(kind=kind, n=_log(rng, 9, 90))
    if kind == "apply":
        return dict(kind=kind, nx=_log(rng, 6, 52), ny=_log(rng, 6, 52), nz=_log(rng, 6, 40),
                    order=rng.choice([1, 2, 2]), rect=rng.random() < 0.7)
    if kind == "xfem":
        order = rng.choice([1, 1, 2])
        return dict(kind=kind, n=_log(rng, 16, 60) if order == 1 else rng.randint(12, 22), order=order,
                    spheres=rng.randint(4, 40), geometry=rng.randint(1, 999))
    if kind == "adjoint":
        return dict(kind=kind, n=rng.randint(20, 42), ncoef=rng.randint(12, 24), order=1,
                    geometry=rng.randint(1, 999))
    if kind == "mgsolve":
        return dict(kind=kind, n=rng.choice([16, 24, 32, 48, 64]))
    return dict(kind=kind, nx=_log(rng, 12, 64), ny=_log(rng, 12, 64))


# --------------------------------------------------------------------------
# inputs
def _mesh(case):
    if case["kind"] in ("plane", "pcg"):
        return mg.hmr_uniform_mesh(2, (case["nx"], case["ny"]), (1.0, case["ny"] / case["nx"]), case.get("order", 1))
    ne = (case["nx"], case["ny"], case["nz"])
    return mg.hmr_uniform_mesh(3, ne, tuple(e / ne[0] for e in ne), case["order"])


def _inputs(case, seed):
    """Everything the model is made of, as host arrays: mesh, sets, u."""
    rng = np.random.default_rng(seed)
    k = case["kind"]
    if k in ("plane", "pcg"):
        mesh = _mesh(case)
        nc, nx = len(mesh["cells"]), case["nx"]
        E = 10.0 ** rng.uniform(-1.0, 0.0, nc)
        left, right = np.arange(0, nc, nx, dtype=np.int32), np.arange(nx - 1, nc, nx, dtype=np.int32)
        sets = [("bulk", dict(ip_cells=np.arange(nc, dtype=np.int32), E=E, rule=mg.RULE_QUAD_2x2)),
                ("dirichlet", dict(cells=left, ordinals=np.full(len(left), 3), E=E[left], rule=mg.RULE_BAR_3)),
                ("neumann", dict(cells=right, ordinals=np.full(len(right), 1), E=E[right], rule=mg.RULE_BAR_3))]
        return dict(dim=2, rect=True, mesh=mesh, sets=sets)
    if k in ("solid", "apply"):
        mesh = _mesh(case)
        nc = len(mesh["cells"])
        if not case["rect"]:
            x = mesh["coords"]
            h, hi = 1.0 / case["nx"], x.max(axis=0)
            inner = np.all((x > 1e-12) & (x < hi - 1e-12), axis=1)
            x[inner] += 0.2 * h * rng.uniform(-1, 1, size=(int(inner.sum()), 3))
        E = 10.0 ** rng.uniform(-3.0, 0.0, nc)
        rule = mg.RULE_HEX_3x3x3 if case["order"] == 2 else mg.RULE_HEX_2x2x2
        return dict(dim=3, rect=case["rect"], mesh=mesh,
                    sets=[("bulk", dict(ip_cells=np.arange(nc, dtype=np.int32), E=E, rule=rule))])
    n = case["n"]
    mesh = mg.hmr_uniform_mesh(3, (n, n, n), (1.0, 1.0, 1.0), 1)
    nc = len(mesh["cells"])
    rho = workloads.smooth_density(n, int(seed))
    cells = np.arange(nc)
    left = cells[cells % n == 0].astype(np.int32)
    right = cells[cells % n == n - 1].astype(np.int32)
    Es = rho[mesh["cells"]].mean(axis=1) ** 3
    sets = [("bulk", dict(ip_cells=cells.astype(np.int32), E=np.ones(nc), rule=mg.RULE_HEX_2x2x2, rho=rho)),
            ("dirichlet", dict(cells=left, ordinals=np.full(len(left), 3), E=Es[left], rule=mg.RULE_QUAD_2x2)),
            ("neumann", dict(cells=right, ordinals=np.full(len(right), 1), E=Es[right], rule=mg.RULE_QUAD_2x2))]
    return dict(dim=3, rect=True, mesh=mesh, sets=sets)


def _stream(m):
    m.set_stream(torch.cuda.current_stream().cuda_stream)


def _build(inp):
    dim = inp["dim"]
    m = mg.FemModel(dim, inp["mesh"], mg.SHAPE_RECTANGULAR if inp["rect"] else mg.SHAPE_GENERAL)
    _stream(m)
    model = mg.MODEL_3D if dim == 3 else mg.MODEL_PLANE_STRAIN
    for kind, a in inp["sets"]:
        if kind == "bulk":
            m.add_bulk_set(a["ip_cells"], a["E"], NU, a["rule"], model, node_density=a.get("rho"))
        elif kind == "dirichlet":
            m.add_side_set(mg.IWG_STRUC_LINEAR_DIRICHLET_SYMMETRIC_NITSCHE, a["cells"], a["ordinals"], a["E"], NU,
                           a["rule"], model, alpha=workloads.NITSCHE_ALPHA, value=(0.0,) * dim)
        else:
            m.add_side_set(mg.IWG_STRUC_LINEAR_NEUMANN, a["cells"], a["ordinals"], a["E"], NU, a["rule"], model,
                           value=(workloads.TRACTION,) + (0.0,) * (dim - 1))
    m.finalize()
    return m


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda")


def _xfem_inputs(case, seed):
    """The level set is the case's (it decides the output sizes), the moduli the seed's."""
    phi = workloads.sphere_field(case["n"], case["geometry"], case["spheres"])
    x = xtk.decompose((case["n"],) * 3, (1.0, 1.0, 1.0), case["order"], phi, device=True)
    E = np.where(x["cell_phase"] == 0, *workloads.XFEM_E) * \
        10.0 ** np.random.default_rng([int(seed), 3]).uniform(-1.0, 0.0, len(x["cell_phase"]))
    sets = workloads.xfem_sets(x)
    for kind, a in sets:
        if kind == "bulk":
            a["E"] = E[a["ip_cells"]]
        else:
            a["EL"], a["EF"] = E[a["leader"]], E[a["follower"]]
    return x, sets


def _adjoint_model(case):
    g = case["geometry"]
    p = sensitivity.levelset_coefficients(case["ncoef"], seed=g, sphere_seed=g + 1, nspheres=12, rmin=0.06, rmax=0.15)
    return sensitivity.build(case["n"], case["ncoef"], case["order"], p=p,
                             stream=torch.cuda.current_stream().cuda_stream)


def _adofs(num, seed):
    # displacement-like values: a dominant smooth part would cancel in the
    # strains, so plain uniform noise is the harder input
    return torch.as_tensor(np.random.default_rng([int(seed), 5]).uniform(-0.5, 0.5, num), device="cuda")


def prepare(case, seed):
    k = case["kind"]
    if k == "xfem":
        x, sets = _xfem_inputs(case, seed)
        m = mg.FemModel(3, x["mesh"], mg.SHAPE_RECTANGULAR)
        _stream(m)
        workloads.add_xfem_sets(m, sets)
        m.finalize()
    elif k == "adjoint":
        c = _adjoint_model(case)
        m = c["model"]
        lam = _adofs(m.num_adofs, seed + 1)
        return dict(kind=k, c=c, u=_adofs(m.num_adofs, seed), lam=lam)
    else:
        m = _build(_inputs(case, seed))
    if k in ("mgsolve", "pcg"):
        rp, ci, vals, b = learned.assembled_system(m)
        multigrid.fcg_config(1, 200)
        return dict(kind=k, m=m, rp=rp, ci=ci, vals=vals, b=b)
    u = _adofs(m.num_adofs, seed)
    s = dict(kind=k, m=m, u=u, rhs=torch.empty_like(u))
    if k != "apply" and case.get("jacobian", True):
        s["vals"] = torch.empty(m.nnz, dtype=F64, device="cuda")
    return s


def run(s):
    k = s["kind"]
    if k in ("plane", "solid", "simp"):
        if "vals" in s:
            s["m"].assemble(s["u"], s["vals"], s["rhs"])
            return dict(vals=s["vals"], rhs=s["rhs"])
        s["m"].assemble(s["u"], None, s["rhs"], mg.NO_JACOBIAN)
        return dict(rhs=s["rhs"])
    if k == "apply":
        s["m"].apply(s["u"], s["rhs"])
        return dict(y=s["rhs"])
    if k == "xfem":
        s["m"].assemble_batched(s["u"], s["vals"], s["rhs"])
        return dict(vals=s["vals"], rhs=s["rhs"])
    if k == "adjoint":
        G, dqdp = sensitivity.sensitivities(s["c"], s["u"], s["lam"])
        return dict(G=G, dqdp=dqdp)
    x = torch.zeros_like(s["b"])
    if k == "mgsolve":
        h = multigrid.Multigrid(s["m"], s["rp"], s["ci"], s["vals"])
        multigrid.fcg_mg(s["m"], s["rp"], s["ci"], s["vals"], s["b"], x, h, rel_tol=1e-8, max_iter=500)
        h.close()
    else:
        s["m"].pcg(s["rp"], s["ci"], s["vals"], s["b"], x, rel_tol=1e-10, max_iter=20000)
    return dict(x=x)


def work(case):
    """Inputs read once (coordinates, material, u), outputs written once."""
    k = case["kind"]
    if k in ("plane", "pcg"):
        d, p, ne = 2, case.get("order", 1), [case["nx"], case["ny"]]
    elif k in ("solid", "apply"):
        d, p, ne = 3, case["order"], [case["nx"], case["ny"], case["nz"]]
    else:
        d, p, ne = 3, case.get("order", 1), [case["n"]] * 3
    cells, nodes, rows, nnz = 1, 1, d, d * d
    for e in ne:
        cells *= e
        nodes *= e + 1
        rows *= e + p
        nnz *= (e + p) * (2 * p + 1) - p * (p + 1)
    vec, geo = 8 * rows, 8 * cells + 8 * d * nodes
    if k in ("plane", "simp", "xfem") or (k == "solid" and case["jacobian"]):
        # every nonzero is a sum of at least one product
        return dict(bytes=8 * nnz + 2 * vec + geo, flops=2 * nnz)
    if k in ("solid", "apply"):
        return dict(bytes=2 * vec + geo, flops=2 * 24 * 24 * cells)
    if k == "adjoint":
        # cells cut by the spheres: a few per cent, 24 tets each, 4 points
        return dict(bytes=2 * vec + 8 * nodes, flops=0.05 * cells * 24 * 4 * 160)
    # solves: the operator read once per iteration and once per smoothing sweep
    its = 12 if k == "mgsolve" else 4 * max(case["nx"], case["ny"])
    return dict(bytes=its * 12 * nnz, flops=2 * its * nnz)


# --------------------------------------------------------------------------
# 64-bit values in plain torch
_S = torch.tensor([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1], [-1, -1, 1], [1, -1, 1], [1, 1, 1],
                   [-1, 1, 1]], dtype=F64)
_FACES = {2: [[0, 1], [1, 2], [2, 3], [3, 0]],
          3: [[1, 5, 4, 0], [1, 2, 6, 5], [3, 7, 6, 2], [0, 4, 7, 3], [0, 3, 2, 1], [4, 5, 6, 7]]}
_G2 = 1.0 / math.sqrt(3.0)
_G3 = math.sqrt(0.6)


def _lagrange(xi):
    """N [..., npe], dN [..., D, npe] of QUAD4 / HEX8 at xi [..., D]."""
    D = xi.shape[-1]
    s = _S[:2 ** D, :D].to(xi.device)
    f = 1.0 + xi.unsqueeze(-2) * s  # [..., npe, D]
    N = f.prod(-1) / 2 ** D
    dN = []
    for i in range(D):
        o = [d for d in range(D) if d != i]
        dN.append(s[:, i] * f[..., o].prod(-1) / 2 ** D)
    return N, torch.stack(dN, -2)


def _gauss(points, dim, dev):
    if points == 2:
        x, w = [-_G2, _G2], [1.0, 1.0]
    else:
        x, w = [-_G3, 0.0, _G3], [5 / 9, 8 / 9, 5 / 9]
    x, w = torch.tensor(x, dtype=F64, device=dev), torch.tensor(w, dtype=F64, device=dev)
    xs = torch.cartesian_prod(*[x] * dim).reshape(-1, dim)
    ws = torch.cartesian_prod(*[w] * dim).reshape(-1, dim).prod(-1)
    return xs, ws


# the 7-point rule of degree 5 and the 4-point tetrahedron rule of degree 2
def _tri7(dev):
    r = math.sqrt(15.0)
    a, b = (6 - r) / 21, (6 + r) / 21
    pts = [[1 / 3, 1 / 3]] + [[p, p] for p in (a, b)] + [[1 - 2 * p, p] for p in (a, b)] + [[p, 1 - 2 * p] for p in
                                                                                           (a, b)]
    wa, wb = (155 - r) / 1200, (155 + r) / 1200
    return torch.tensor(pts, dtype=F64, device=dev), torch.tensor([9 / 40] + [wa, wb] * 3, dtype=F64, device=dev)


def _tet4(dev):
    a, b = (5 - math.sqrt(5.0)) / 20, (5 + 3 * math.sqrt(5.0)) / 20
    pts = [[a, a, a], [b, a, a], [a, b, a], [a, a, b]]
    return torch.tensor(pts, dtype=F64, device=dev), torch.full((4,), 0.25, dtype=F64, device=dev)


def _tet_n(z):
    # TET4 node order: xi_0, xi_1, 1 - sum, xi_2
    return torch.stack([z[..., 0], z[..., 1], 1 - z.sum(-1), z[..., 2]], -1)


def _grads(X, xi):
    """N [n|1,q,npe], g [n,q,D,npe] = dN/dx, det J [n,q] of the cells X [n,npe,D]."""
    N, dN = _lagrange(xi)
    if dN.dim() == 3:
        N, dN = N.unsqueeze(0), dN.unsqueeze(0)
    J = torch.einsum("nqia,naj->nqij", dN.expand(X.shape[0], *dN.shape[1:]), X)
    return N, torch.linalg.solve(J, dN.expand(X.shape[0], *dN.shape[1:])), torch.linalg.det(J)


def _lame(E):
    return E * NU / ((1 + NU) * (1 - 2 * NU)), E / (2 * (1 + NU))


def _bulk_k(g, w):
    """w = w* E [n,q]: K [n,npe,npe,D,D] (node pair, field pair)."""
    A = torch.einsum("nqia,nqjb->nabij", g * w[..., None, None], g)
    lam, mu = _lame(1.0)
    K = lam * A + mu * A.transpose(-1, -2)
    tr = mu * A.diagonal(dim1=-2, dim2=-1).sum(-1)
    return K + tr[..., None, None] * torch.eye(g.shape[-2], dtype=F64, device=g.device)


def _traction(g, n, E):
    """t_f = T[..., f, g, b] u_gb: g [n,q,D,npe], n [n,q,D], E [n]."""
    lam, mu = _lame(E)
    D = n.shape[-1]
    e = torch.eye(D, dtype=F64, device=n.device)
    T = lam[:, None, None, None, None] * torch.einsum("nqf,nqgb->nqfgb", n, g)
    m = torch.einsum("nqg,nqfb->nqfgb", n, g) + torch.einsum("fg,nqk,nqkb->nqfgb", e, n, g)
    return T + mu[:, None, None, None, None] * m


def _facet(fx, xq):
    """w-free measure and normal of facets with vertices fx [n,nv,D] at facet points xq [q,D-1]."""
    nv, D = fx.shape[1:]
    if nv == 3:
        N = torch.stack([xq[:, 0], xq[:, 1], 1 - xq.sum(-1)], -1)
        dN = torch.tensor([[1.0, 0.0, -1.0], [0.0, 1.0, -1.0]], dtype=F64, device=fx.device).expand(len(xq), 2, 3)
    elif nv == 2:
        N = torch.stack([(1 - xq[:, 0]) / 2, (1 + xq[:, 0]) / 2], -1)
        dN = torch.tensor([[-0.5, 0.5]], dtype=F64, device=fx.device).expand(len(xq), 1, 2)
    else:
        N, dN = _lagrange(xq)
    t = torch.einsum("qma,nad->nqmd", dN, fx)
    if D == 2:
        c = torch.stack([t[..., 0, 1], -t[..., 0, 0]], -1)
    else:
        c = torch.linalg.cross(t[..., 0, :], t[..., 1, :])
    det = c.norm(dim=-1)
    return N, det * (0.5 if nv == 3 else 1.0), c / det[..., None]


class _System:
    """Node-level operator collected pair by pair, projected on the spline bases."""

    def __init__(self, mesh, used_cells, dim, u):
        dev = "cuda"
        self.dim, self.npe = dim, 2 ** dim
        self.cells = _dev(mesh["cells"]).long()
        self.X = _dev(mesh["coords"])
        off, tb, tw = _dev(mesh["t_off"]), _dev(mesh["t_bases"]).long(), _dev(mesh["t_w"])
        self.nn = len(off) - 1
        cnt = off[1:] - off[:-1]
        self.wid = int(cnt.max())
        # extraction rows padded to one width with weight 0 (basis of the first entry)
        idx = off[:-1, None] + torch.minimum(torch.arange(self.wid, device=dev)[None], cnt[:, None] - 1)
        tbp = tb[idx]
        self.w = torch.where(torch.arange(self.wid, device=dev)[None] < cnt[:, None], tw[idx], torch.zeros_like(tw[idx]))
        mark = torch.zeros(int(mesh["num_bases"]), dtype=torch.long, device=dev)
        nodes = self.cells[used_cells].reshape(-1).unique()
        mark[tbp[nodes].reshape(-1)] = 1
        rank = mark.cumsum(0) - 1
        self.nu = int(mark.sum())
        self.b = rank[tbp]
        self.un = torch.einsum("nk,nkf->nf", self.w, u.reshape(dim, self.nu).T[self.b.clamp(min=0)]) if u is not None \
            else None
        self.keys, self.vals = [], []
        self.r = torch.zeros(self.nn, dim, dtype=F64, device=dev)

    def add(self, nodes, K, R=None):
        """nodes [n,m], K [n,m,m,D,D] or None, R [n,m,D] (default K u)."""
        if K is not None:
            self.keys.append((nodes[:, :, None] * self.nn + nodes[:, None, :]).reshape(-1))
            self.vals.append(K.reshape(-1, self.dim ** 2))
            if R is None:
                R = torch.einsum("nabfg,nbg->naf", K, self.un[nodes])
            if len(self.keys) > 6:
                self._fold()
        self.r.index_add_(0, nodes.reshape(-1), R.reshape(-1, self.dim))

    def _fold(self):
        k, inv = torch.cat(self.keys).unique(return_inverse=True)
        v = torch.zeros(len(k), self.dim ** 2, dtype=F64, device=k.device)
        v.index_add_(0, inv, torch.cat(self.vals))
        self.keys, self.vals = [k], [v]

    def rhs(self):
        out = torch.zeros(self.nu, self.dim, dtype=F64, device=self.r.device)
        for k in range(self.wid):
            ok = self.w[:, k] != 0
            out.index_add_(0, self.b[ok, k], self.r[ok] * self.w[ok, k, None])
        return out.T.reshape(-1).contiguous()

    def csr(self):
        self._fold()
        key, v, D = self.keys[0], self.vals[0], self.dim
        n, m = key // self.nn, key % self.nn
        pair = lambda i, j: self.b[n, i] * self.nu + self.b[m, j]  # noqa: E731
        uniq = None
        for i in range(self.wid):
            part = torch.cat([pair(i, j) for j in range(self.wid)])
            uniq = part.unique() if uniq is None else torch.cat([uniq, part.unique()]).unique()
        row = uniq // self.nu
        ulen = torch.bincount(row, minlength=self.nu)
        start = ulen.cumsum(0) - ulen
        out = torch.zeros(D * D * len(uniq), dtype=F64, device=key.device)
        for i in range(self.wid):
            for j in range(self.wid):
                wij = self.w[n, i] * self.w[m, j]
                at = torch.searchsorted(uniq, pair(i, j))
                r = row[at]
                base = D * start[r] + (at - start[r])
                for f in range(D):
                    for g in range(D):
                        out.index_add_(0, f * D * len(uniq) + base + g * ulen[r], wij * v[:, f * D + g])
        return out


def _exact_sets(inp, u, jacobian):
    D = inp["dim"]
    S = _System(inp["mesh"], slice(None), D, u)
    for kind, a in inp["sets"]:
        cells = _dev(a["ip_cells"] if kind == "bulk" else a["cells"]).long()
        E = _dev(a["E"])
        if kind == "bulk":
            xi, w = _gauss(3 if a["rule"] == mg.RULE_HEX_3x3x3 else 2, D, "cuda")
            rho = None if a.get("rho") is None else _dev(a["rho"])
            for c0 in range(0, len(cells), 32768):
                nd = S.cells[cells[c0:c0 + 32768]]
                N, g, det = _grads(S.X[nd], xi)
                ws = w * det * E[c0:c0 + 32768, None]
                if rho is not None:
                    ws = ws * torch.einsum("nqa,na->nq", N.expand(len(nd), -1, -1), rho[nd]) ** 3
                K = _bulk_k(g, ws)
                S.add(nd, K) if jacobian else S.add(nd, None, torch.einsum("nabfg,nbg->naf", K, S.un[nd]))
            continue
        xq, w = _gauss(3 if D == 2 else 2, D - 1, "cuda")
        nd = S.cells[cells]
        face = torch.tensor(_FACES[D][int(a["ordinals"][0])], device="cuda")
        Nf, meas, n = _facet(S.X[nd[:, face]], xq)
        xi = torch.einsum("qa,ad->qd", Nf, _S[:2 ** D, :D].cuda()[face])
        N, g, _ = _grads(S.X[nd], xi)
        N, ws = N.expand(len(nd), -1, -1), w * meas
        if kind == "neumann":
            t = torch.zeros(D, dtype=F64, device="cuda")
            t[0] = workloads.TRACTION
            S.add(nd, None, -torch.einsum("nq,nqa,f->naf", ws, N, t))
            continue
        h = ws.sum(-1) if D == 2 else torch.sqrt(4 * ws.sum(-1) / math.pi)
        gamma = workloads.NITSCHE_ALPHA * E / h
        T = _traction(g, n, E)
        K = -torch.einsum("nq,nqgfa,nqb->nabfg", ws, T, N) - torch.einsum("nq,nqa,nqfgb->nabfg", ws, N, T)
        NN = torch.einsum("nq,nqa,nqb->nab", ws, N, N) * gamma[:, None, None]
        K = K + NN[..., None, None] * torch.eye(D, dtype=F64, device="cuda")
        S.add(nd, K) if jacobian else S.add(nd, None, torch.einsum("nabfg,nbg->naf", K, S.un[nd]))
    return S


def _exact_xfem(x, sets, u):
    used = torch.cat([_dev(a["ip_cells"] if k == "bulk" else np.concatenate([a["leader"], a["follower"]])).long()
                      for k, a in sets])
    S = _System(x["mesh"], used, 3, u)
    vol = torch.zeros(len(S.cells), dtype=F64, device="cuda")
    tz, tw = _tet4("cuda")
    for kind, a in sets:
        if kind != "bulk":
            continue
        cells, E = _dev(a["ip_cells"]).long(), _dev(a["E"])
        if a.get("ig_offsets") is None:
            xi, w = _gauss(2, 3, "cuda")
            for c0 in range(0, len(cells), 65536):
                nd = S.cells[cells[c0:c0 + 65536]]
                _, g, det = _grads(S.X[nd], xi)
                S.add(nd, _bulk_k(g, w * det * E[c0:c0 + 65536, None]))
            continue
        off = _dev(a["ig_offsets"]).long()
        item = torch.repeat_interleave(torch.arange(len(cells), device="cuda"), off[1:] - off[:-1])
        tx, tp = _dev(a["ig_coords"]).reshape(-1, 4, 3), _dev(a["ig_param"]).reshape(-1, 4, 3)
        det = torch.linalg.det(tx[:, [0, 1, 3]] - tx[:, 2:3]) / 6
        vol.index_add_(0, cells[item], det.abs())
        for t0 in range(0, len(item), 65536):
            sl = slice(t0, t0 + 65536)
            nd = S.cells[cells[item[sl]]]
            _, g, _ = _grads(S.X[nd], torch.einsum("qk,nkd->nqd", _tet_n(tz), tp[sl]))
            S.add(nd, _bulk_k(g, tw * (det * E[item])[sl, None]))
    for kind, a in sets:
        if kind == "bulk":
            continue
        off = _dev(a["offsets"]).long()
        item = torch.repeat_interleave(torch.arange(len(off) - 1, device="cuda"), off[1:] - off[:-1])
        sides = [_dev(a["leader"]).long(), _dev(a["follower"]).long()]
        Es = [_dev(a["EL"]), _dev(a["EF"])]
        iface = a["iwg"] == mg.IWG_STRUC_LINEAR_INTERFACE_SYMMETRIC_NITSCHE
        nv = 3 if iface else 4
        fx = _dev(a["coords"]).reshape(-1, nv, 3)
        fp = [_dev(a["leader_param"]).reshape(-1, nv, 3), _dev(a["follower_param"]).reshape(-1, nv, 3)]
        xq, w = _tri7("cuda") if iface else _gauss(2, 2, "cuda")
        area = torch.zeros(len(off) - 1, dtype=F64, device="cuda")
        Nf, meas, n = _facet(fx, xq)
        area.index_add_(0, item, (w * meas).sum(-1))
        eye = torch.eye(3, dtype=F64, device="cuda")
        for f0 in range(0, len(item), 32768):
            sl = slice(f0, f0 + 32768)
            it, ws, nq = item[sl], w * meas[sl], n[sl]
            nds, Ns, gs, Ts = [], [], [], []
            for s in (0, 1):
                nd = S.cells[sides[s][it]]
                N, g, _ = _grads(S.X[nd], torch.einsum("qk,nkd->nqd", Nf, fp[s][sl]))
                nds.append(nd), Ns.append(N), gs.append(g), Ts.append(_traction(g, nq, Es[s][it]))
            nd = torch.cat(nds, 1)
            if iface:
                v = [vol[sides[s][it]] / Es[s][it] for s in (0, 1)]
                wt = [v[0] / (v[0] + v[1]), v[1] / (v[0] + v[1])]
                gamma = 2 * a["alpha"] * area[it] / (v[0] + v[1])
                jump = torch.cat([Ns[0], -Ns[1]], 2)                                     # [u] = jump . u
                mean = torch.cat([Ts[s] * wt[s][:, None, None, None, None] for s in (0, 1)], 4)  # {t}
                K = -torch.einsum("nq,nqa,nqfgb->nabfg", ws, jump, mean)
                K = K - torch.einsum("nq,nqgfa,nqb->nabfg", ws, mean, jump)
                JJ = torch.einsum("nq,nqa,nqb->nab", ws * gamma[:, None], jump, jump)
                K = K + JJ[..., None, None] * eye
            else:
                # virtual-work ghost: the jump of the stress against the jump of
                # the n-projected test strain
                e = []
                for g in gs:
                    ng = torch.einsum("nqk,nqka->nqa", nq, g)
                    off_ = torch.einsum("nqf,nqha->nqhfa", nq, g)
                    d = ng[:, :, None] - nq[..., None] * g
                    e.append(off_ + torch.einsum("nqha,hf->nqhfa", d, eye))
                eps = torch.cat([e[0], -e[1]], 4)
                tj = torch.cat([Ts[0], -Ts[1]], 4)
                h = torch.sqrt(4 * area[it] / math.pi) * a["alpha"]
                K = torch.einsum("nq,nqhfa,nqhgb->nabfg", ws * h[:, None], eps, tj)
            S.add(nd, K)
    return S


def _exact_adjoint(case, seed):
    c = _adjoint_model(case)
    x, sets, m = c["x"], c["sets"], c["model"]
    u, lam = _adofs(m.num_adofs, seed), _adofs(m.num_adofs, seed + 1)
    used = torch.cat([_dev(a["ip_cells"] if k != "double" else np.concatenate([a["leader"], a["follower"]])).long()
                      for k, a in sets])
    S, Sl = _System(x["mesh"], used, 3, u), _System(x["mesh"], used, 3, lam)
    v = x["vertices"]
    kind, par, xv, val = _dev(v["kind"]), _dev(v["parents"]).long(), _dev(v["coords"]), _dev(v["value"])
    mov = torch.nonzero(kind == 3)[:, 0]
    t = val[mov].clone().requires_grad_(True)
    p0, p1 = xv[par[mov, 0]], xv[par[mov, 1]]
    pos = xv.clone().index_copy(0, mov, p0 + t[:, None] * (p1 - p0))
    lame = _lame(1.0)

    def stress(G):
        tr = G.diagonal(dim1=-2, dim2=-1).sum(-1)
        return lame[0] * tr[..., None, None] * torch.eye(3, dtype=F64, device="cuda") + lame[1] * (G + G.transpose(-1, -2))

    def fields(cells, pts):
        nd = S.cells[cells]
        X0, X6 = S.X[nd[:, 0]], S.X[nd[:, 6]]
        N, dN = _lagrange(-1 + 2 * (pts - X0[:, None]) / (X6 - X0)[:, None])
        g = dN * (2 / (X6 - X0))[:, None, :, None]
        return [(torch.einsum("nqa,naf->nqf", N, q.un[nd]), torch.einsum("nqia,naf->nqfi", g, q.un[nd]))
                for q in (S, Sl)]

    vol = torch.zeros(len(S.cells), dtype=F64, device="cuda")
    F = torch.zeros((), dtype=F64, device="cuda")
    tz, tw = _tet4("cuda")
    for k, a in sets:
        if k != "bulk" or a.get("ig_offsets") is None:
            continue
        off = _dev(a["ig_offsets"]).long()
        cell = torch.repeat_interleave(_dev(a["ip_cells"]).long(), off[1:] - off[:-1])
        E = torch.repeat_interleave(_dev(a["E"]), off[1:] - off[:-1])
        tx = pos[_dev(a["ig_vertex_ids"]).long().reshape(-1, 4)]
        e = tx[:, [0, 1, 3]] - tx[:, 2:3]
        det = (torch.linalg.cross(e[:, 0], e[:, 1]) * e[:, 2]).sum(-1) / 6
        vol = vol.index_add(0, cell, det.abs())
        (_, Gu), (_, Gl) = fields(cell, torch.einsum("qk,nkd->nqd", _tet_n(tz), tx))
        phi = (stress(Gu) * (0.5 * Gu - Gl)).sum((-1, -2))
        F = F + (tw * phi * (det * E)[:, None]).sum()
    for k, a in sets:
        if k != "double" or a["iwg"] != mg.IWG_STRUC_LINEAR_INTERFACE_SYMMETRIC_NITSCHE:
            continue
        off = _dev(a["offsets"]).long()
        item = torch.repeat_interleave(torch.arange(len(off) - 1, device="cuda"), off[1:] - off[:-1])
        fx = pos[_dev(a["facet_vertex_ids"]).long().reshape(-1, 3)]
        xq, w = _tri7("cuda")
        cr = torch.linalg.cross(fx[:, 0] - fx[:, 2], fx[:, 1] - fx[:, 2])
        nn = cr.norm(dim=-1)
        n, ws = cr / nn[:, None], w * (0.5 * nn)[:, None]
        area = torch.zeros(len(off) - 1, dtype=F64, device="cuda").index_add(0, item, ws.sum(-1))
        pts = torch.einsum("qk,nkd->nqd", torch.stack([xq[:, 0], xq[:, 1], 1 - xq.sum(-1)], -1), fx)
        sides, Es = [_dev(a["leader"]).long(), _dev(a["follower"]).long()], [_dev(a["EL"]), _dev(a["EF"])]
        vE = [vol[sides[s]] / Es[s] for s in (0, 1)]
        wt = [(vE[s] / (vE[0] + vE[1]))[item] for s in (0, 1)]
        gamma = (2 * a["alpha"] * area / (vE[0] + vE[1]))[item]
        fl = [fields(sides[s][item], pts) for s in (0, 1)]
        ju, jl = fl[0][0][0] - fl[1][0][0], fl[0][1][0] - fl[1][1][0]
        tr = [sum(torch.einsum("nqij,nj->nqi", stress(fl[s][q][1]), n) * (wt[s] * Es[s][item])[:, None, None]
                  for s in (0, 1)) for q in (0, 1)]
        dens = -(jl * tr[0]).sum(-1) - (tr[1] * ju).sum(-1) + gamma[:, None] * (jl * ju).sum(-1)
        F = F - (ws * dens).sum()
    G = torch.zeros(len(kind), dtype=F64, device="cuda")
    G[mov] = torch.autograd.grad(F, t)[0]
    # t = f0 / (f0 - f1), a parent's level set the mean of its background nodes
    f0, f1 = val[par[mov, 0]], val[par[mov, 1]]
    dt = [-f1 / (f0 - f1) ** 2, f0 / (f0 - f1) ** 2]
    cols, tm = _dev(c["cols"]).long(), _dev(c["vals"])
    dqdp = torch.zeros(len(c["p"]), dtype=F64, device="cuda")
    count = torch.tensor([1, 4, 8], device="cuda")
    for k in (0, 1):
        q = par[mov, k]
        cn = count[kind[q].long()]
        for j in range(8):
            ok = j < cn
            nd = par[q[ok], j]
            dqdp.index_add_(0, cols[nd].reshape(-1), (tm[nd] * (G[mov] * dt[k] / cn)[ok, None]).reshape(-1))
    return dict(G=G, dqdp=dqdp)


def exact(case, seed):
    k = case["kind"]
    if k in ("mgsolve", "pcg"):
        return None  # an iterate: its distance from the solution is the stopping tolerance's, not rounding's
    if k == "adjoint":
        return _exact_adjoint(case, seed)
    if k == "xfem":
        x, sets = _xfem_inputs(case, seed)
        m = x["mesh"]
        cells = np.concatenate([a["ip_cells"] if q == "bulk" else np.concatenate([a["leader"], a["follower"]])
                                for q, a in sets])
        nodes = np.unique(m["cells"][np.unique(cells)])
        mark = np.zeros(int(m["num_bases"]), dtype=bool)
        for j in range(int((m["t_off"][1:] - m["t_off"][:-1]).max())):
            at = m["t_off"][nodes] + j
            mark[m["t_bases"][at[at < m["t_off"][nodes + 1]]]] = True
        S = _exact_xfem(x, sets, _adofs(3 * int(mark.sum()), seed))
        return dict(vals=S.csr(), rhs=S.rhs())
    inp = _inputs(case, seed)
    D = inp["dim"]
    if k == "plane":
        num = D * (case["nx"] + case["order"]) * (case["ny"] + case["order"])
    elif k == "simp":
        num = D * (case["n"] + 1) ** 3
    else:
        num = D * (case["nx"] + case["order"]) * (case["ny"] + case["order"]) * (case["nz"] + case["order"])
    jac = k != "apply" and case.get("jacobian", True)
    S = _exact_sets(inp, _adofs(num, seed), jac)
    if k == "apply":
        return dict(y=S.rhs())
    return dict(vals=S.csr(), rhs=S.rhs()) if jac else dict(rhs=S.rhs())
