"""Brick kernels of the XFEM clusters (fem_brick.cu) against the oracle: every
kind of equation object, alone and mixed with objects that the classification
leaves to the general cluster kernel.

The tolerance is the parity tests': 1e-12 per CSR row.  An entry is a sum of
at most a few hundred products of comparable size, so its rounding stays below
1e3 * 2^-53 = 1.1e-13 of the row's largest term."""
import numpy as np
import pytest

import moris_gb300 as mg
from moris_gb300 import workloads, xtk
from tests.common import RTOL, csr_row_rel_err, rel_err, uniform01

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    t = pytest.importorskip("torch")
    if not t.cuda.is_available():
        pytest.skip("no CUDA device")
    return t


def _grade(x, mesh):
    """Cells of unequal size: every coordinate mapped by t -> t (1 + t) / 2 on
    the mesh, the facets and the integration cells (which stay inside their
    cells; parametric coordinates recomputed from the corners)."""
    f = lambda c: 0.5 * c * (1.0 + c)  # noqa: E731
    mesh["coords"] = f(mesh["coords"])
    X0, X6 = mesh["coords"][mesh["cells"][:, 0]], mesh["coords"][mesh["cells"][:, 6]]
    par = lambda c, p: -1.0 + 2.0 * (p - X0[c][:, None]) / (X6 - X0)[c][:, None]  # noqa: E731
    for k in (0, 1):
        c = x["cut%d" % k]
        item = np.repeat(c["cells"], np.diff(c["ig_offsets"]))
        pts = f(c["ig_coords"]).reshape(-1, 4, 3)
        c["ig_coords"], c["ig_param"] = pts.ravel(), par(item, pts).ravel()
        g = x["ghost%d" % k]
        g["coords"] = f(g["coords"])
    i = x["interface"]
    pts = f(i["coords"]).reshape(-1, 3, 3)
    i["coords"] = pts.ravel()
    i["param"] = par(np.repeat(i["leader"], np.diff(i["offsets"])), pts).ravel()


def _perturb(x, mesh):
    """Some objects the brick kernels refuse, some with another vertex order."""
    tw, off = mesh["t_w"], mesh["t_off"]
    for n in range(0, len(off) - 1, 37):
        tw[off[n]:off[n + 1]] *= 1.0 + 1e-3 * (1 + n % 5)
    for k in (0, 1):
        g = x["ghost%d" % k]
        arr = [g[a].reshape(-1, 4, 3) for a in ("coords", "leader_param", "follower_param")]
        for a in arr:
            a[1::3] = np.roll(a[1::3], 1, axis=1)       # another first corner
            a[2::3] = a[2::3, ::-1].copy()              # opposite normal
        # every fifth facet in two halves (two facets of one cluster)
        out, offs = [[], [], []], [0]
        for i in range(len(arr[0])):
            for a, o in zip(arr, out):
                if i % 5:
                    o.append(a[i:i + 1])
                else:
                    m = 0.5 * (a[i, [0, 1]] + a[i, [3, 2]])
                    o.append(np.stack([np.concatenate([a[i, :2], m[::-1]]), np.concatenate([m, a[i, 2:]])]))
            offs.append(offs[-1] + len(out[0][-1]))
        for name, o in zip(("coords", "leader_param", "follower_param"), out):
            g[name] = np.concatenate(o).ravel()
        g["offsets"] = np.array(offs, dtype=np.int64)


@pytest.mark.parametrize("mixed", [False, True], ids=["bricks", "mixed"])
@pytest.mark.parametrize("ghost", [mg.IWG_STRUC_LINEAR_VW_GHOST, mg.IWG_GHOST_NORMAL_FIELD], ids=["vw", "normal"])
@pytest.mark.parametrize("order,n,rule,tri", [(1, 7, mg.RULE_TET_4, mg.RULE_TRI_7), (2, 4, mg.RULE_TET_4, mg.RULE_TRI_7),
                                              (1, 5, mg.RULE_TET_11, mg.RULE_TRI_3)])
def test_xfem_clusters_match_oracle(torch, order, n, rule, tri, ghost, mixed):
    from oracle import OracleModel
    x = xtk.decompose((n, n, n), (1.0, 1.0, 1.0), order, workloads.sphere_field(n, 17, 3, 0.2, 0.33))
    mesh = x["mesh"]
    _grade(x, mesh)
    if mixed:
        _perturb(x, mesh)
    sets = workloads.xfem_sets(x, tet_rule=rule, tri_rule=tri, ghost_iwg=ghost)
    Ec = 0.2 + uniform01(9, len(mesh["cells"]))
    for kind, a in sets:
        if kind == "bulk":
            a["E"] = Ec[a["ip_cells"]]
        else:
            a["EL"], a["EF"] = Ec[a["leader"]], Ec[a["follower"]]
            if mixed and a["facet_cell"] == mg.CELL_TRI3:
                a["iwg"] = mg.IWG_STRUC_LINEAR_INTERFACE_UNSYMMETRIC_NITSCHE
    prod = mg.FemModel(3, mesh, mg.SHAPE_RECTANGULAR)
    workloads.add_xfem_sets(prod, sets)
    prod.set_stream(torch.cuda.current_stream().cuda_stream)
    prod.finalize()
    orc = OracleModel(3, mg.CELL_HEX8, mg.SHAPE_RECTANGULAR, mesh)
    for kind, a in sets:
        if kind == "bulk":
            orc.add_bulk_set(a["ig_cell"], a["rule"], mg.MODEL_3D, a["ip_cells"], a["E"], a["nu"], a.get("ig_offsets"),
                             a.get("ig_coords"), a.get("ig_param"))
    for kind, a in sets:
        if kind == "double":
            orc.add_double_side_set(a["iwg"], a["facet_cell"], a["rule"], mg.MODEL_3D, a["leader"], a["follower"],
                                    a["offsets"], a["coords"], a["leader_param"], a["follower_param"], a["EL"],
                                    a["EF"], a["nu"], a["alpha"])
    orc.finalize()
    un = uniform01(4, prod.num_adofs) - 0.5
    vo, ro = orc.assemble(un)
    rp, _ = prod.graph()
    u = torch.tensor(un, device="cuda")
    vals = torch.full((prod.nnz,), float("nan"), dtype=torch.float64, device="cuda")
    rhs = torch.full((prod.num_adofs,), float("nan"), dtype=torch.float64, device="cuda")

    def check(scale=1.0):
        assert csr_row_rel_err(rp, vals.cpu().numpy(), scale * vo) <= RTOL
        assert rel_err(rhs.cpu().numpy(), scale * ro) <= RTOL

    prod.assemble_batched(u, vals, rhs)
    check()
    prod.assemble_batched(u, vals, rhs, mg.ACCUMULATE)  # the same buffers, no zero fill
    check(2.0)
    prod.assemble(u, vals, rhs)
    check()
    rhs.fill_(float("nan"))
    prod.assemble_batched(u, vals, rhs, mg.NO_JACOBIAN)
    check()
    vals.fill_(float("nan"))
    prod.assemble_batched(None, vals, rhs, mg.NO_RESIDUAL)
    check()
    vh, rh = prod.assemble_host(un)
    assert csr_row_rel_err(rp, vh, vo) <= RTOL and rel_err(rh, ro) <= RTOL


@pytest.mark.parametrize("iwg", [mg.IWG_STRUC_LINEAR_NEUMANN, mg.IWG_STRUC_LINEAR_DIRICHLET_SYMMETRIC_NITSCHE,
                                 mg.IWG_STRUC_LINEAR_DIRICHLET_UNSYMMETRIC_NITSCHE])
@pytest.mark.parametrize("ordinal", range(6))
def test_boundary_facets_match_oracle(torch, iwg, ordinal):
    """Every facet of a brick, unequal edges, prescribed value and thickness."""
    from oracle import OracleModel
    mesh = mg.hmr_uniform_mesh(3, (3, 2, 4), (1.0, 0.7, 1.9), 1)
    mesh["coords"][:, 2] *= 0.5 + mesh["coords"][:, 2]
    nc = len(mesh["cells"])
    cells = np.arange(nc, dtype=np.int32)
    E = uniform01(6, nc) + 0.2
    prod = mg.FemModel(3, mesh, mg.SHAPE_RECTANGULAR)
    orc = OracleModel(3, mg.CELL_HEX8, mg.SHAPE_RECTANGULAR, mesh)
    prod.add_bulk_set(cells, E, 0.3, mg.RULE_HEX_2x2x2, mg.MODEL_3D)
    orc.add_bulk_set(mg.CELL_HEX8, mg.RULE_HEX_2x2x2, mg.MODEL_3D, cells, E, 0.3)
    some, val = cells[::2], (0.02, -0.01, 0.03)
    prod.add_side_set(iwg, some, np.full(len(some), ordinal), E[some], 0.25, mg.RULE_QUAD_2x2, mg.MODEL_3D, alpha=20.0,
                      value=val, thickness=0.8)
    orc.add_side_set(iwg, mg.RULE_QUAD_2x2, mg.MODEL_3D, some, np.full(len(some), ordinal), E[some], 0.25, 20.0, val)
    orc.set_side_options(0, 0.8, None)
    prod.finalize()
    orc.finalize()
    un = uniform01(8, prod.num_adofs) - 0.5
    rp, _ = prod.graph()
    vals = torch.empty(prod.nnz, dtype=torch.float64, device="cuda")
    rhs = torch.empty(prod.num_adofs, dtype=torch.float64, device="cuda")
    for u in (un, np.zeros_like(un)):
        vo, ro = orc.assemble(u)
        prod.assemble(torch.tensor(u, device="cuda") if u is un else None, vals, rhs)
        assert csr_row_rel_err(rp, vals.cpu().numpy(), vo) <= RTOL
        assert rel_err(rhs.cpu().numpy(), ro) <= RTOL
