"""Side sets that share launches (four per launch) against the oracle: six sets of
different size and kind on one model, after a lattice and after the element loop."""
import numpy as np
import pytest

import moris_gb300 as mg
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
