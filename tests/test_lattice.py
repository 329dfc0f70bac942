"""Tensor-lattice assembly (fem_lattice.cu) against the oracle and against the
element loop, at the edges of its tiles (8 x 4 x 4 nodes, 8 x 4 bases).

The tolerance is the parity tests': 1e-12 per CSR row.  Every value is a sum
of at most 64 products, so its rounding is below 64 * 2^-53 = 7e-15 of the
row's largest term."""
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


def _assemble(torch, m, u, flags=0, vals=None, rhs=None):
    vals = torch.full((m.nnz,), float("nan"), dtype=torch.float64, device="cuda") if vals is None else vals
    rhs = torch.full((m.num_adofs,), float("nan"), dtype=torch.float64, device="cuda") if rhs is None else rhs
    torch.cuda.synchronize()
    m.assemble(u, None if flags & mg.NO_JACOBIAN else vals, None if flags & mg.NO_RESIDUAL else rhs, flags)
    return vals, rhs


# quadratic splines below 1,024 cells are assembled by the element loop
SIZES = [(1, 1, 1), (2, 1, 3), (7, 3, 3), (8, 4, 4), (6, 2, 3), (9, 5, 2), (17, 6, 5), (4, 16, 16), (17, 9, 7)]


@pytest.mark.parametrize("density", [False, True], ids=["E", "rho"])
@pytest.mark.parametrize("p,rule", [(1, mg.RULE_HEX_2x2x2), (1, mg.RULE_HEX_3x3x3), (2, mg.RULE_HEX_2x2x2),
                                    (2, mg.RULE_HEX_3x3x3)])
@pytest.mark.parametrize("ne", SIZES, ids=lambda n: "x".join(map(str, n)))
def test_lattice_assembly_matches_oracle_and_element_loop(torch, ne, p, rule, density):
    prod, orc, _ = problem(3, ne, p, mg.SHAPE_RECTANGULAR, rule, sides=True, density=density)
    prod.finalize()
    orc.finalize()
    un = uniform01(31, prod.num_adofs) - 0.5
    u = torch.tensor(un, device="cuda")
    rp, _ = prod.graph()
    vo, ro = orc.assemble(un, nthreads=4)
    vals, rhs = _assemble(torch, prod, u)
    assert csr_row_rel_err(rp, vals.cpu().numpy(), vo) <= RTOL
    assert rel_err(rhs.cpu().numpy(), ro) <= RTOL
    # one output alone, no u, and sums on top of values that are there
    assert torch.equal(_assemble(torch, prod, u, mg.NO_RESIDUAL)[0], vals) or \
        csr_row_rel_err(rp, _assemble(torch, prod, u, mg.NO_RESIDUAL)[0].cpu().numpy(), vo) <= RTOL
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


@pytest.mark.parametrize("p", [1, 2])
@pytest.mark.parametrize("ne", [(1, 2, 1), (8, 3, 5), (13, 12, 12)], ids=lambda n: "x".join(map(str, n)))
def test_lattice_apply_and_several_sets(torch, ne, p):
    """Two sets over the same cells in another order, graded cells, the
    matrix-free product and a non-finite modulus product's status."""
    mesh = mg.hmr_uniform_mesh(3, ne, (1.0, 0.7, 1.3), p)
    x = mesh["coords"]
    x[:, 0] = x[:, 0] ** 2 + 0.1 * x[:, 0]  # graded along x: still a tensor lattice
    nc = len(mesh["cells"])
    order = np.random.default_rng(2).permutation(nc).astype(np.int32)
    E1, E2 = uniform01(3, nc) + 0.1, uniform01(4, nc) + 0.1
    out = []
    for pin in (False, True):
        m = mg.FemModel(3, mesh, mg.SHAPE_RECTANGULAR)
        m.add_bulk_set(order, E1, 0.3, mg.RULE_HEX_3x3x3, mg.MODEL_3D)
        m.add_bulk_set(np.arange(nc, dtype=np.int32), E2, 0.0, mg.RULE_HEX_2x2x2, mg.MODEL_3D)
        m.finalize()
        if pin:
            m.set_variant(0, 2)
            m.set_variant(1, 2)
        u = torch.tensor(uniform01(5, m.num_adofs) - 0.5, device="cuda")
        vals, rhs = _assemble(torch, m, u)
        y = torch.full_like(u, float("nan"))
        m.apply(u, y)
        y2 = y.clone()
        m.apply(u, y2, mg.ACCUMULATE)
        torch.cuda.synchronize()
        out.append([t.cpu().numpy() for t in (vals, rhs, y, y2)])
    rp, _ = m.graph()
    assert csr_row_rel_err(rp, out[0][0], out[1][0]) <= RTOL
    for a, b in zip(out[0][1:], out[1][1:]):
        assert rel_err(a, b) <= RTOL
    assert rel_err(out[0][2], out[0][1]) <= RTOL and rel_err(out[0][3], 2 * out[0][2]) <= RTOL


def test_rows_of_a_large_linear_lattice(torch):
    """From 65,536 nodes on, constant moduli go through the stencil as well (density
    sets always do): against the element loop, and summed onto values that are there."""
    prod, _, _ = problem(3, (41, 40, 38), 1, mg.SHAPE_RECTANGULAR, mg.RULE_HEX_2x2x2)
    prod.finalize()
    u = torch.tensor(uniform01(31, prod.num_adofs) - 0.5, device="cuda")
    vals, rhs = _assemble(torch, prod, u)
    v2, r2 = _assemble(torch, prod, u, mg.ACCUMULATE, vals.clone(), rhs.clone())
    prod.set_variant(0, 2)
    vg, rg = _assemble(torch, prod, u)
    rp, _ = prod.graph()
    assert csr_row_rel_err(rp, vals.cpu().numpy(), vg.cpu().numpy()) <= RTOL
    assert csr_row_rel_err(rp, v2.cpu().numpy(), 2 * vg.cpu().numpy()) <= RTOL
    assert rel_err(rhs.cpu().numpy(), rg.cpu().numpy()) <= RTOL and rel_err(r2.cpu().numpy(), 2 * rg.cpu().numpy()) <= RTOL


def test_non_finite_blocks_are_reported(torch):
    """A modulus whose products overflow: both paths return the status."""
    for p in (1, 2):
        mesh = mg.hmr_uniform_mesh(3, (3, 2, 2), (1e-3, 1.0, 1.0), p)
        for pin in (False, True):
            m = mg.FemModel(3, mesh, mg.SHAPE_RECTANGULAR)
            m.add_bulk_set(np.arange(12, dtype=np.int32), np.full(12, 1e308), 0.49, mg.RULE_HEX_2x2x2, mg.MODEL_3D)
            m.finalize()
            if pin:
                m.set_variant(0, 2)
            with pytest.raises(mg.FemGpuError) as e:
                _assemble(torch, m, None)
            assert e.value.status == 3


@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("ne", [(1, 1), (2, 3), (5, 1), (31, 2), (7, 33)], ids=lambda n: "x".join(map(str, n)))
def test_plane_lattice_matches_oracle_and_element_loop(torch, ne, p):
    prod, orc, _ = problem(2, ne, p, mg.SHAPE_RECTANGULAR, mg.RULE_QUAD_2x2, sides=True)
    prod.finalize()
    orc.finalize()
    un = uniform01(37, prod.num_adofs) - 0.5
    u = torch.tensor(un, device="cuda")
    rp, _ = prod.graph()
    vo, ro = orc.assemble(un)
    vals, rhs = _assemble(torch, prod, u)
    assert csr_row_rel_err(rp, vals.cpu().numpy(), vo) <= RTOL
    assert rel_err(rhs.cpu().numpy(), ro) <= RTOL
    assert rel_err(_assemble(torch, prod, u, mg.NO_JACOBIAN)[1].cpu().numpy(), ro) <= RTOL
    v2, r2 = _assemble(torch, prod, u, mg.ACCUMULATE, vals.clone(), rhs.clone())
    assert csr_row_rel_err(rp, v2.cpu().numpy(), 2 * vo) <= RTOL and rel_err(r2.cpu().numpy(), 2 * ro) <= RTOL
    prod.set_variant(0, 2)
    vg, rg = _assemble(torch, prod, u)
    assert csr_row_rel_err(rp, vals.cpu().numpy(), vg.cpu().numpy()) <= RTOL
    assert rel_err(rhs.cpu().numpy(), rg.cpu().numpy()) <= RTOL


@pytest.mark.parametrize("p", [1, 2, 3])
def test_plane_stress_graded_lattice(torch, p):
    """Plane stress, graded cells, cells in another order, matrix-free product."""
    mesh = mg.hmr_uniform_mesh(2, (9, 6), (1.0, 0.7), p)
    x = mesh["coords"]
    x[:, 1] = x[:, 1] ** 2 + 0.2 * x[:, 1]
    nc = len(mesh["cells"])
    order = np.random.default_rng(2).permutation(nc).astype(np.int32)
    out = []
    for pin in (False, True):
        m = mg.FemModel(2, mesh, mg.SHAPE_RECTANGULAR)
        m.add_bulk_set(order, uniform01(3, nc) + 0.1, 0.2, mg.RULE_QUAD_2x2, mg.MODEL_PLANE_STRESS)
        m.finalize()
        if pin:
            m.set_variant(0, 2)
        u = torch.tensor(uniform01(5, m.num_adofs) - 0.5, device="cuda")
        vals, rhs = _assemble(torch, m, u)
        y = torch.full_like(u, float("nan"))
        m.apply(u, y)
        torch.cuda.synchronize()
        out.append([t.cpu().numpy() for t in (vals, rhs, y)])
    rp, _ = m.graph()
    assert csr_row_rel_err(rp, out[0][0], out[1][0]) <= RTOL
    assert rel_err(out[0][1], out[1][1]) <= RTOL and rel_err(out[0][2], out[1][2]) <= RTOL
