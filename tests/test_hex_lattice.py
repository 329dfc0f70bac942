"""Cells of any shape on a tensor lattice of nodes (fem_hex.cuh) against the oracle
and the element loop, around the cells per CTA and the tiles of the projection.

Tolerance as in the parity tests, 1e-12 per CSR row: sums of at most 8 x 27 products
of factors that themselves carry the rounding of one 3 x 3 inverse (cond < 10)."""
import numpy as np
import pytest

import moris_gb300 as mg
from tests.common import RTOL, csr_row_rel_err, distort, problem, rel_err, uniform01

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    t = pytest.importorskip("torch")
    if not t.cuda.is_available():
        pytest.skip("no CUDA device")
    return t


def _assemble(torch, m, u, flags=0, vals=None, rhs=None):
    vals = torch.full((m.nnz,), float("nan"), dtype=torch.float64, device="cuda") if vals is None else vals
    rhs = torch.full((m.num_adofs,), float("nan"), dtype=torch.float64, device="cuda") if rhs is None else rhs
    torch.cuda.synchronize()
    m.assemble(u, None if flags & mg.NO_JACOBIAN else vals, None if flags & mg.NO_RESIDUAL else rhs, flags)
    return vals, rhs


@pytest.mark.parametrize("p,rule", [(1, mg.RULE_HEX_2x2x2), (1, mg.RULE_HEX_3x3x3), (2, mg.RULE_HEX_2x2x2),
                                    (2, mg.RULE_HEX_3x3x3)])
@pytest.mark.parametrize("ne", [(1, 1, 1), (2, 1, 3), (5, 4, 1), (7, 3, 6), (3, 19, 18), (32, 2, 16)], ids=lambda n: "x".join(map(str, n)))
def test_distorted_lattice_matches_oracle_and_element_loop(torch, ne, p, rule):
    prod, orc, _ = problem(3, ne, p, mg.SHAPE_GENERAL, rule, sides=True)
    prod.finalize()
    orc.finalize()
    un = uniform01(31, prod.num_adofs) - 0.5
    u = torch.tensor(un, device="cuda")
    rp, _ = prod.graph()
    vo, ro = orc.assemble(un, nthreads=4)
    vals, rhs = _assemble(torch, prod, u)
    assert csr_row_rel_err(rp, vals.cpu().numpy(), vo) <= RTOL
    assert rel_err(rhs.cpu().numpy(), ro) <= RTOL
    assert csr_row_rel_err(rp, _assemble(torch, prod, u, mg.NO_RESIDUAL)[0].cpu().numpy(), vo) <= RTOL
    assert rel_err(_assemble(torch, prod, u, mg.NO_JACOBIAN)[1].cpu().numpy(), ro) <= RTOL
    f0 = orc.assemble(np.zeros_like(un))[1]
    assert rel_err(_assemble(torch, prod, None, mg.NO_JACOBIAN)[1].cpu().numpy(), f0) <= RTOL
    v2, r2 = _assemble(torch, prod, u, mg.ACCUMULATE, vals.clone(), rhs.clone())
    assert csr_row_rel_err(rp, v2.cpu().numpy(), 2 * vo) <= RTOL and rel_err(r2.cpu().numpy(), 2 * ro) <= RTOL
    # the element loop on the same model
    prod.set_variant(0, 2)
    vg, rg = _assemble(torch, prod, u)
    assert csr_row_rel_err(rp, vals.cpu().numpy(), vg.cpu().numpy()) <= RTOL
    assert rel_err(rhs.cpu().numpy(), rg.cpu().numpy()) <= RTOL
    # the matrix-free product (bulk sets only) by the lattice and by the element loop
    bulk, _, _ = problem(3, ne, p, mg.SHAPE_GENERAL, rule)
    bulk.finalize()
    y, z = torch.full_like(u, float("nan")), torch.full_like(u, float("nan"))
    bulk.apply(u, y)
    bulk.set_variant(0, 2)
    bulk.apply(u, z)
    torch.cuda.synchronize()
    assert rel_err(y.cpu().numpy(), z.cpu().numpy()) <= RTOL


@pytest.mark.parametrize("p", [1, 2])
def test_other_order_and_inverted_cells(torch, p):
    """A set in another order keeps the element loop; points of negative volume are
    skipped on both paths, so that mirrored cells assemble to zero."""
    ne = (4, 3, 2)
    mesh = distort(mg.hmr_uniform_mesh(3, ne, [1.0] * 3, p), 3, ne, 0.2, 9)
    nc = len(mesh["cells"])
    E = uniform01(3, nc) + 0.1

    def run(order, pin):
        m = mg.FemModel(3, mesh, mg.SHAPE_GENERAL)
        m.add_bulk_set(order, E[order], 0.3, mg.RULE_HEX_2x2x2, mg.MODEL_3D)
        m.finalize()
        if pin:
            m.set_variant(0, 2)
        u = torch.tensor(uniform01(5, m.num_adofs) - 0.5, device="cuda")
        return m.graph()[0], [t.cpu().numpy() for t in _assemble(torch, m, u)]

    natural = np.arange(nc, dtype=np.int32)
    rp, a = run(natural, False)
    _, b = run(np.random.default_rng(2).permutation(nc).astype(np.int32), False)
    assert csr_row_rel_err(rp, a[0], b[0]) <= RTOL and rel_err(a[1], b[1]) <= RTOL
    mesh["coords"] = mesh["coords"] * np.array([-1.0, 1.0, 1.0])
    for pin in (False, True):
        _, c = run(natural, pin)
        assert not c[0].any() and not c[1].any()
