"""Side sets that share launches (four per launch) against the oracle: six sets of
different size and kind on one model, after a lattice and after the element loop."""
import numpy as np
import pytest

import moris_gb300 as mg
from oracle import OracleModel
from tests.common import RTOL, csr_row_rel_err, problem, rel_err, uniform01

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    t = pytest.importorskip("torch")
    if not t.cuda.is_available():
        pytest.skip("no CUDA device")
    return t


@pytest.mark.parametrize("dim,ne,p", [(2, (9, 7), 1), (2, (9, 7), 2), (2, (70, 33), 3), (3, (3, 2, 4), 2),
                                      (3, (11, 10, 10), 2)])
@pytest.mark.parametrize("shape", [mg.SHAPE_RECTANGULAR, mg.SHAPE_GENERAL], ids=["bricks", "distorted"])
def test_six_side_sets(torch, dim, ne, p, shape):
    prod, orc, mesh = problem(dim, ne, p, shape, sides=True)
    nc = len(mesh["cells"])
    c = np.arange(nc)
    rule = mg.RULE_BAR_3 if dim == 2 else mg.RULE_QUAD_2x2
    model = mg.MODEL_PLANE_STRAIN if dim == 2 else mg.MODEL_3D
    row = c // ne[0] % ne[1]
    zero, load = (0.0,) * dim, (2e-3,) * dim
    for k, (cells, ordinal) in enumerate([(c[row == 0], 0), (c[row == ne[1] - 1], 2), (c[row == 0][:1], 0),
                                          (c[row == ne[1] - 1][::2], 2)]):
        cells = cells.astype(np.int32)
        o, E = np.full(len(cells), ordinal), 0.1 + uniform01(40 + k, len(cells))
        if k % 2 == 0:
            iwg = mg.IWG_STRUC_LINEAR_DIRICHLET_SYMMETRIC_NITSCHE
            prod.add_side_set(iwg, cells, o, E, 0.3, rule, model, alpha=50.0, value=zero)
            orc.add_side_set(iwg, rule, model, cells, o, E, 0.3, 50.0, zero)
        else:
            iwg = mg.IWG_STRUC_LINEAR_NEUMANN
            prod.add_side_set(iwg, cells, o, E, 0.3, rule, model, value=load)
            orc.add_side_set(iwg, rule, model, cells, o, E, 0.3, 0.0, load)
    prod.finalize()
    orc.finalize()
    un = uniform01(31, prod.num_adofs) - 0.5
    vals = torch.full((prod.nnz,), float("nan"), dtype=torch.float64, device="cuda")
    rhs = torch.full((prod.num_adofs,), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    prod.assemble(torch.tensor(un, device="cuda"), vals, rhs)
    vo, ro = orc.assemble(un, nthreads=4)
    assert csr_row_rel_err(prod.graph()[0], vals.cpu().numpy(), vo) <= RTOL
    assert rel_err(rhs.cpu().numpy(), ro) <= RTOL


@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("ne", [(1, 1), (1, 6), (13, 2)], ids=lambda n: "x".join(map(str, n)))
def test_plane_lattice_facets(torch, ne, p):
    """All four sides of a plane lattice: both Nitsche signs with a prescribed value,
    plane stress, thickness, the one-point rule, and a set with a Select matrix, which
    keeps the general kernel; against the oracle, with and without u."""
    mesh = mg.hmr_uniform_mesh(2, ne, [1.3, 0.6], p)
    nc = len(mesh["cells"])
    prod = mg.FemModel(2, mesh, mg.SHAPE_RECTANGULAR)
    orc = OracleModel(2, mg.CELL_QUAD4, mg.SHAPE_RECTANGULAR, mesh)
    cells, E = np.arange(nc, dtype=np.int32), 0.1 + uniform01(3, nc)
    prod.add_bulk_set(cells, E, 0.3, mg.RULE_QUAD_2x2, mg.MODEL_PLANE_STRESS)
    orc.add_bulk_set(mg.CELL_QUAD4, mg.RULE_QUAD_2x2, mg.MODEL_PLANE_STRESS, cells, E, 0.3)
    c = np.arange(nc)
    x, y = c % ne[0], c // ne[0]
    sym, uns, neu = (mg.IWG_STRUC_LINEAR_DIRICHLET_SYMMETRIC_NITSCHE, mg.IWG_STRUC_LINEAR_DIRICHLET_UNSYMMETRIC_NITSCHE,
                     mg.IWG_STRUC_LINEAR_NEUMANN)
    select = np.diag([1.0, 0.0])
    sides = [(c[x == 0], 3, sym, mg.RULE_BAR_3, (0.3, -0.2), 1.0, None),
             (c[x == ne[0] - 1], 1, uns, mg.RULE_BAR_3, (0.1, 0.4), 0.7, None),
             (c[y == 0], 0, neu, mg.RULE_BAR_3, (0.5, -1.5), 1.0, None),
             (c[y == ne[1] - 1], 2, sym, mg.RULE_BAR_1, (0.0, 0.25), 1.6, None),
             (c[y == ne[1] - 1], 2, sym, mg.RULE_BAR_3, (0.2, 0.1), 1.0, select)]
    for k, (cl, o, iwg, rule, value, thick, sel) in enumerate(sides):
        cl = cl.astype(np.int32)
        Es = 0.1 + uniform01(50 + k, len(cl))
        prod.add_side_set(iwg, cl, np.full(len(cl), o), Es, 0.25, rule, mg.MODEL_PLANE_STRESS, alpha=20.0, value=value,
                          thickness=thick, select=sel)
        orc.add_side_set(iwg, rule, mg.MODEL_PLANE_STRESS, cl, np.full(len(cl), o), Es, 0.25, 20.0, value)
        orc.set_side_options(k, thick, sel)
    prod.finalize()
    orc.finalize()
    for un in (uniform01(31, prod.num_adofs) - 0.5, None):
        vals = torch.full((prod.nnz,), float("nan"), dtype=torch.float64, device="cuda")
        rhs = torch.full((prod.num_adofs,), float("nan"), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        prod.assemble(None if un is None else torch.tensor(un, device="cuda"), vals, rhs)
        vo, ro = orc.assemble(np.zeros(prod.num_adofs) if un is None else un)
        assert csr_row_rel_err(prod.graph()[0], vals.cpu().numpy(), vo) <= RTOL
        assert rel_err(rhs.cpu().numpy(), ro) <= RTOL
