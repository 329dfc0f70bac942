"""Adjoint sensitivities of an interface whose leader and follower are
different cells of unequal size: the follower's field polynomials are moved to
the leader's centre (fem_sensitivity.cu).  G against central differences of
Q - lambda^T R in the edge coordinate.

Tolerance: central differences with h = 1e-5 of a smooth function of t of order
one have a truncation error near h^2 = 1e-10 and a rounding error near
2^-53 |F| / h = 1e-11 |F| per unit of G; 1e-7 leaves room for |F| / |G| = 1e3."""
import numpy as np
import pytest

import moris_gb300 as mg
from moris_gb300 import sensitivity
from tests.common import uniform01

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("rule", [(mg.RULE_TET_4, mg.RULE_TRI_7), (mg.RULE_TET_11, mg.RULE_TRI_3)])
def test_interface_between_different_cells(order, rule):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    mesh = mg.hmr_uniform_mesh(3, (2, 1, 1), (1.0, 0.8, 0.9), order)
    X = mesh["coords"]
    X[X[:, 0] > 0.9, 0] = 1.3  # the second cell is longer
    cells = mesh["cells"]
    nn = len(X)
    # IG vertices: the background nodes, the cells' centres, two moving ones on
    # the diagonals of the shared face and of an outer face of the second cell
    faces = [[1, 5, 4, 0], [1, 2, 6, 5], [3, 7, 6, 2], [0, 4, 7, 3], [0, 3, 2, 1], [4, 5, 6, 7]]
    shared = [cells[0][k] for k in faces[1]]   # corners A, B, C, D
    outer = [cells[1][k] for k in faces[5]]
    kind = np.array([0] * nn + [2, 2, 3, 3], dtype=np.int32)
    par = np.zeros((nn + 4, 8), dtype=np.int32)
    par[:nn, 0] = np.arange(nn)
    par[nn], par[nn + 1] = cells[0], cells[1]
    par[nn + 2, :2], par[nn + 3, :2] = shared[::2], outer[::2]
    t = np.zeros(nn + 4)
    t[nn + 2:] = 0.4, 0.63

    def place(tv):
        x = np.concatenate([X, X[cells].mean(axis=1)[:2], np.zeros((2, 3))])
        for v in (nn + 2, nn + 3):
            x[v] = x[par[v, 0]] + tv[v] * (x[par[v, 1]] - x[par[v, 0]])
        return x

    x = place(t)
    fan = lambda q, v: [(q[i], q[(i + 1) % 4], v) for i in range(4)]  # noqa: E731

    def tets(c):
        out = []
        for f in faces:
            q = [cells[c][k] for k in f]
            if set(q) == set(shared):
                tri = fan(q, nn + 2)
            elif c == 1 and set(q) == set(outer):
                tri = fan(q, nn + 3)
            else:
                tri = [(q[0], q[1], q[2]), (q[0], q[2], q[3])]
            for a, b, d in tri:
                # TET4 order with a positive volume: edges from the third vertex
                p = [a, b, nn + c, d]
                e = [x[p[k]] - x[p[2]] for k in (0, 1, 3)]
                out.append(p if np.dot(e[0], np.cross(e[1], e[2])) > 0 else [b, a, nn + c, d])
        return np.array(out, dtype=np.int32)

    par_of = lambda c, y: -1.0 + 2.0 * (y - X[cells[c][0]]) / (X[cells[c][6]] - X[cells[c][0]])  # noqa: E731
    m = mg.FemModel(3, mesh, mg.SHAPE_RECTANGULAR)
    for c in (0, 1):
        tv = tets(c)
        m.add_bulk_set([c], [1.0 - 0.4 * c], 0.3, rule[0], mg.MODEL_3D, ig_cell=mg.CELL_TET4,
                       ig_offsets=[0, len(tv)], ig_coords=x[tv].ravel(), ig_param=par_of(c, x[tv]).ravel(),
                       ig_vertex_ids=tv)
    tri = np.array(fan(shared, nn + 2), dtype=np.int32)
    m.add_double_side_set(mg.IWG_STRUC_LINEAR_INTERFACE_SYMMETRIC_NITSCHE, [0], [1], [0, len(tri)], x[tri].ravel(),
                          par_of(0, x[tri]).ravel(), par_of(1, x[tri]).ravel(), [1.0], [0.6], 0.3, rule[1],
                          mg.CELL_TRI3, 10.0, facet_vertex_ids=tri)
    m.set_stream(torch.cuda.current_stream().cuda_stream)
    m.set_ig_vertices(kind, par, x, t)
    m.finalize()
    u = torch.tensor(uniform01(3, m.num_adofs) - 0.5, device="cuda")
    lam = torch.tensor(uniform01(4, m.num_adofs) - 0.5, device="cuda")
    G = torch.empty(nn + 4, dtype=torch.float64, device="cuda")
    m.drdp_adjoint(u, lam, G)
    g = G.cpu().numpy()
    assert np.all(g[:nn + 2] == 0)
    h = 1e-5
    for v in (nn + 2, nn + 3):
        f = []
        for s in (1.0, -1.0):
            tt = t.copy()
            tt[v] += s * h
            m.update_ig_vertices(tt)
            f.append(sensitivity.functional(m, u, lam))
        m.update_ig_vertices(t)
        fd = (f[0] - f[1]) / (2 * h)
        assert abs(fd - g[v]) <= 1e-7 * max(abs(g[v]), abs(f[0])), (v, fd, g[v])
