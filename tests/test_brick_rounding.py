"""Rounding of the brick kernels (fem_brick.cu): batched assembly of a small level-set model
against the same weak forms in extended precision, with the library's own rule constants.

The bound is on the 2-norm of the error over that of the values, in units of roundoff
(2^-53).  A value is a product of about ten rounded factors (1.8 units if each adds
1/sqrt(3) of one) and a sum of some twenty moments and terms, which adds about half a unit
as long as the terms are of one size and no sum runs over more than twenty in a row."""
import numpy as np
import pytest

import moris_gb300 as mg
from moris_gb300 import workloads, xtk

L = np.longdouble
pytestmark = [pytest.mark.gpu, pytest.mark.skipif(np.finfo(L).eps > 1e-18, reason="no extended precision")]
NU = L(workloads.XFEM_NU)
S = np.array([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1], [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]], L)
EYE = np.eye(3, dtype=L)


def _gauss(dim):
    x = np.array([-0.577350269189626, 0.577350269189626], dtype=L)
    g = np.stack(np.meshgrid(*[x] * dim, indexing="ij"), -1).reshape(-1, dim)
    return g, np.ones(len(g), dtype=L)


def _tri7():
    a, b, c, d, t = 0.797426985353087, 0.101286507323456, 0.059715871789770, 0.470142064105115, 0.333333333333333
    p = [[t, t], [a, b], [b, a], [b, b], [c, d], [d, c], [d, d]]
    return np.array(p, dtype=L), np.array([0.225] + [0.125939180544827] * 3 + [0.132394152788506] * 3, dtype=L)


def _shape(xi, s):
    f = 1 + xi[..., None, :] * s
    D = s.shape[1]
    dN = [s[:, i] * f[..., [d for d in range(D) if d != i]].prod(-1) / 2 ** D for i in range(D)]
    return f.prod(-1) / 2 ** D, np.stack(dN, -2)


def _lame(E):
    return E * NU / ((1 + NU) * (1 - 2 * NU)), E / (2 * (1 + NU))


def _cells(X, xi):
    N, dN = _shape(xi, S)
    N, dN = (N, dN) if N.ndim == 3 else (N[None], dN[None])
    J = (X[:, 6] - X[:, 0]) / 2
    return N, dN / J[:, None, :, None], J.prod(-1)[:, None]


def _bulk(g, w):
    A = np.einsum("nqia,nqjb->nabij", g * w[..., None, None], np.broadcast_to(g, w.shape + g.shape[2:]))
    lam, mu = _lame(L(1))
    return lam * A + mu * A.swapaxes(-1, -2) + (mu * np.trace(A, axis1=-2, axis2=-1))[..., None, None] * EYE


def _traction(g, n, E):
    lam, mu = (c[:, None, None, None, None] for c in _lame(E))
    m = np.einsum("nqg,nqfb->nqfgb", n, g) + np.einsum("fg,nqk,nqkb->nqfgb", EYE, n, g)
    return lam * np.einsum("nqf,nqgb->nqfgb", n, g) + mu * m


def _facets(fx, xq):
    if fx.shape[1] == 3:
        N = np.stack([xq[:, 0], xq[:, 1], 1 - xq.sum(-1)], -1)
        dN, half = np.broadcast_to(np.array([[1, 0, -1], [0, 1, -1]], dtype=L), (len(xq), 2, 3)), L(0.5)
    else:
        (N, dN), half = _shape(xq, S[:4, :2]), L(1)
    t = np.einsum("qma,nad->nqmd", dN, fx)
    c = np.cross(t[..., 0, :], t[..., 1, :])
    det = np.sqrt((c * c).sum(-1))
    return N, det * half, c / det[..., None]


def _double(a, mesh, vol):
    """Node lists and matrices of an interface or ghost set, a facet each."""
    item = np.repeat(np.arange(len(a["offsets"]) - 1), np.diff(a["offsets"]))
    iface = a["iwg"] == mg.IWG_STRUC_LINEAR_INTERFACE_SYMMETRIC_NITSCHE
    fx = a["coords"].reshape(-1, 3 if iface else 4, 3).astype(L)
    xq, w = _tri7() if iface else _gauss(2)
    Nf, meas, n = _facets(fx, xq)
    ws, area = w * meas, np.zeros(len(a["offsets"]) - 1, dtype=L)
    np.add.at(area, item, ws.sum(-1))
    area, nd, N, g, T, v = area[item], [], [], [], [], []
    for cells, xi, E in ((a["leader"], a["leader_param"], a["EL"]), (a["follower"], a["follower_param"], a["EF"])):
        c, E = cells[item], E[item].astype(L)
        nd.append(mesh["cells"][c])
        Ns, gs, _ = _cells(mesh["coords"].astype(L)[nd[-1]], np.einsum("qk,nkd->nqd", Nf, xi.reshape(fx.shape).astype(L)))
        N.append(Ns), g.append(gs), T.append(_traction(gs, n, E)), v.append(vol[c] / E)
    if iface:
        jump = np.concatenate([N[0], -N[1]], 2)
        mean = np.concatenate([T[s] * (v[s] / (v[0] + v[1]))[:, None, None, None, None] for s in (0, 1)], 4)
        gamma = 2 * L(a["alpha"]) * area / (v[0] + v[1])
        K = -np.einsum("nq,nqa,nqfgb->nabfg", ws, jump, mean) - np.einsum("nq,nqgfa,nqb->nabfg", ws, mean, jump)
        K = K + np.einsum("nq,nqa,nqb->nab", ws * gamma[:, None], jump, jump)[..., None, None] * EYE
    else:
        e = []
        for q in g:
            d = np.einsum("nqk,nqka->nqa", n, q)[:, :, None] - n[..., None] * q
            e.append(np.einsum("nqf,nqha->nqhfa", n, q) + np.einsum("nqha,hf->nqhfa", d, EYE))
        h = L(a["alpha"]) * np.sqrt(4 * area / L("3.14159265358979323846264338327950288"))
        eps = np.concatenate([e[0], -e[1]], 4) * (ws * h[:, None])[:, :, None, None, None]
        K = np.einsum("nqhfa,nqhgb->nabfg", eps, np.concatenate([T[0], -T[1]], 4))
    return np.concatenate(nd, 1), K


def _values(mesh, sets):
    """CSR values (columns of a row ascending, rows and columns component-major)."""
    X, vol, nodes, mats = mesh["coords"].astype(L), np.zeros(len(mesh["cells"]), dtype=L), [], []
    a, b = 0.585410196624968, 0.138196601125010
    z = np.array([[a, b, b], [b, a, b], [b, b, a], [b, b, b]], dtype=L)
    tet = np.stack([z[:, 0], z[:, 1], 1 - z.sum(-1), z[:, 2]], -1)
    for kind, s in sets:
        if kind != "bulk":
            continue
        nd, E = mesh["cells"][s["ip_cells"]], s["E"].astype(L)
        if s.get("ig_offsets") is None:
            xi, w = _gauss(3)
            _, g, det = _cells(X[nd], xi)
            nodes.append(nd), mats.append(_bulk(g, w * det * E[:, None]))
            continue
        item = np.repeat(np.arange(len(E)), np.diff(s["ig_offsets"]))
        tx = s["ig_coords"].reshape(-1, 4, 3).astype(L)
        e = tx[:, [0, 1, 3]] - tx[:, 2:3]
        det = (np.cross(e[:, 0], e[:, 1]) * e[:, 2]).sum(-1) / 6
        np.add.at(vol, s["ip_cells"][item], np.abs(det))
        _, g, _ = _cells(X[nd[item]], np.einsum("qk,nkd->nqd", tet, s["ig_param"].reshape(-1, 4, 3).astype(L)))
        nodes.append(nd[item]), mats.append(_bulk(g, np.repeat((det * E[item] / 4)[:, None], 4, 1)))
    for kind, s in sets:
        if kind != "bulk":
            nd, K = _double(s, mesh, vol)
            nodes.append(nd), mats.append(K)
    # the bases of a node (width entries each), numbered among the used ones
    width = int(mesh["t_off"][1])
    tb, tw = mesh["t_bases"].reshape(-1, width).astype(np.int64), mesh["t_w"].reshape(-1, width).astype(L)
    rank = np.zeros(int(mesh["num_bases"]), dtype=np.int64)
    for nd in nodes:
        rank[tb[nd].reshape(-1)] = 1
    nu, rank = int(rank.sum()), rank.cumsum() - 1
    nn, keys, vals = len(tb), [], []
    for nd, K in zip(nodes, mats):
        keys.append((nd[:, :, None].astype(np.int64) * nn + nd[:, None, :]).reshape(-1)), vals.append(K.reshape(-1, 9))
    key, at = np.unique(np.concatenate(keys), return_inverse=True)
    v = np.zeros((len(key), 9), dtype=L)
    np.add.at(v, at.reshape(-1), np.concatenate(vals))
    pairs = [(rank[tb[key // nn, i]] * nu + rank[tb[key % nn, j]], tw[key // nn, i] * tw[key % nn, j])
             for i in range(width) for j in range(width)]
    pos = np.unique(np.concatenate([p for p, _ in pairs]))
    out = np.zeros((len(pos), 9), dtype=L)
    for p, w in pairs:
        np.add.at(out, np.searchsorted(pos, p), w[:, None] * v)
    count = np.bincount(pos // nu, minlength=nu)
    rows = np.split(out, count.cumsum()[:-1])
    return np.concatenate([r[:, 3 * f + g] for f in range(3) for r in rows for g in range(3)])


def _part(sets, part):
    """cut: the cut clusters alone.  interface: with cut clusters, which give it its volumes,
    of no stiffness.  all: the whole model."""
    if part == "all":
        return sets
    cut = [(k, a) for k, a in sets if a.get("ig_offsets") is not None]
    if part == "cut":
        return cut
    return [(k, dict(a, E=a["E"] * 1e-40)) for k, a in cut] + \
        [(k, a) for k, a in sets if a.get("iwg") == mg.IWG_STRUC_LINEAR_INTERFACE_SYMMETRIC_NITSCHE]


@pytest.mark.parametrize("order,n,spheres,geometry,part,units", [(1, 9, 4, 3, "cut", 2.5), (2, 5, 2, 5, "cut", 2.5),
                                                               (1, 9, 4, 3, "interface", 2.1), (1, 9, 4, 3, "all", 2.5)])
def test_values_against_extended_precision(order, n, spheres, geometry, part, units):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    phi = workloads.sphere_field(n, geometry, spheres)
    x = xtk.decompose((n,) * 3, (1.0, 1.0, 1.0), order, phi, device=False)
    E = np.where(x["cell_phase"] == 0, *workloads.XFEM_E) * \
        10.0 ** np.random.default_rng(3).uniform(-1.0, 0.0, len(x["cell_phase"]))
    sets = workloads.xfem_sets(x)
    for kind, a in sets:
        if kind == "bulk":
            a["E"] = E[a["ip_cells"]]
        else:
            a["EL"], a["EF"] = E[a["leader"]], E[a["follower"]]
    sets = _part(sets, part)
    m = mg.FemModel(3, x["mesh"], mg.SHAPE_RECTANGULAR)
    workloads.add_xfem_sets(m, sets)
    m.finalize()
    vals = torch.empty(m.nnz, dtype=torch.float64, device="cuda")
    m.assemble_batched(None, vals, None, mg.NO_RESIDUAL)
    ref = _values(x["mesh"], sets)
    assert len(ref) == m.nnz
    err = vals.cpu().numpy().astype(L) - ref
    assert np.sqrt((err * err).sum() / (ref * ref).sum()) <= units * 2.0 ** -53
