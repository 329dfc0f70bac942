"""The lattice kernels (fem_lattice.cu, fem_hex.cuh) at sizes that reach them: models of
at least kLatticeCells cells (fem_internal.hpp), with edges of one to three cells, where
the CSR rows' boxes and the projection's tiles are clipped, and with node and basis counts
on and beside the multiples of their blocks (32 consecutive nodes, 5 x 3 bases).

The tolerance is the parity tests': 1e-12 per CSR row.  Every value is a sum of at most 64
products, so its rounding is below 64 * 2^-53 = 7e-15 of the row's largest term."""
import os
import re

import numpy as np
import pytest

import moris_gb300 as mg
from tests.common import RTOL, csr_row_rel_err, distort, problem, rel_err, uniform01

HEADER = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "moris_gb300", "csrc",
                      "fem_internal.hpp")


def _lines():
    """Cells from which bricks take the lattice: assembly, product of quadratic splines."""
    with open(HEADER) as f:
        text = f.read()
    assembly = re.search(r"kLatticeCells = (\d+);", text).group(1)
    product = re.search(r"quad && product \? (\d+) : kLatticeCells", text).group(1)
    return int(assembly), int(product)


# thin along each axis; 1,331 nodes and 12 x 12 bases; 1,568 = 49 x 32 nodes and 15 x 15
# bases; 16 x 13 bases; 1,440 = 45 x 32 nodes
SIZES = [(1, 32, 33), (33, 1, 32), (32, 33, 1), (2, 23, 24), (19, 18, 3), (10, 10, 10), (13, 13, 7), (14, 11, 7),
         (15, 14, 5)]
PRODUCTS = [(1, 42, 42), (42, 1, 42), (42, 42, 1), (2, 30, 29), (29, 20, 3), (12, 12, 12)]
_ids = lambda n: "x".join(map(str, n))  # noqa: E731


def test_the_sizes_reach_the_lattice():
    assembly, product = _lines()
    assert min(np.prod(n) for n in SIZES) >= assembly and min(np.prod(n) for n in PRODUCTS) >= product


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


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["E", "rho", "distorted"])
@pytest.mark.parametrize("p,rule", [(1, mg.RULE_HEX_2x2x2), (2, mg.RULE_HEX_3x3x3)], ids=["linear", "quadratic"])
@pytest.mark.parametrize("ne", SIZES, ids=_ids)
def test_assembly_matches_oracle(torch, ne, p, rule, kind):
    prod, orc, _ = problem(3, ne, p, mg.SHAPE_GENERAL if kind == "distorted" else mg.SHAPE_RECTANGULAR, rule,
                           density=kind == "rho")
    prod.finalize()
    orc.finalize()
    un = uniform01(31, prod.num_adofs) - 0.5
    u = torch.tensor(un, device="cuda")
    rp, _ = prod.graph()
    vo, ro = orc.assemble(un, nthreads=4)
    before = prod.launch_count()
    vals, rhs = _assemble(torch, prod, u)
    # the element loop is one launch; so are linear splines on the lattice, but for densities
    assert (prod.launch_count() - before > 1) == (p == 2 or kind == "rho")
    assert csr_row_rel_err(rp, vals.cpu().numpy(), vo) <= RTOL
    assert rel_err(rhs.cpu().numpy(), ro) <= RTOL
    assert csr_row_rel_err(rp, _assemble(torch, prod, u, mg.NO_RESIDUAL)[0].cpu().numpy(), vo) <= RTOL
    assert rel_err(_assemble(torch, prod, u, mg.NO_JACOBIAN)[1].cpu().numpy(), ro) <= RTOL
    assert not _assemble(torch, prod, None, mg.NO_JACOBIAN)[1].any()
    v2, r2 = _assemble(torch, prod, u, mg.ACCUMULATE, vals.clone(), rhs.clone())
    assert csr_row_rel_err(rp, v2.cpu().numpy(), 2 * vo) <= RTOL and rel_err(r2.cpu().numpy(), 2 * ro) <= RTOL


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["E", "rho", "distorted"])
@pytest.mark.parametrize("p", [1, 2])
@pytest.mark.parametrize("ne", PRODUCTS, ids=_ids)
def test_products_match_the_element_loop(torch, ne, p, kind):
    m, _, _ = problem(3, ne, p, mg.SHAPE_GENERAL if kind == "distorted" else mg.SHAPE_RECTANGULAR,
                      mg.RULE_HEX_2x2x2, density=kind == "rho")
    m.finalize()
    u = torch.tensor(uniform01(5, m.num_adofs) - 0.5, device="cuda")
    y, z = torch.full_like(u, float("nan")), torch.full_like(u, float("nan"))
    before = m.launch_count()
    m.apply(u, y)
    assert (m.launch_count() - before > 1) == (p == 2 or kind == "rho")
    y2 = y.clone()
    m.apply(u, y2, mg.ACCUMULATE)
    m.set_variant(0, 2)
    m.apply(u, z)
    torch.cuda.synchronize()
    assert rel_err(y.cpu().numpy(), z.cpu().numpy()) <= RTOL
    assert rel_err(y2.cpu().numpy(), 2 * z.cpu().numpy()) <= RTOL


def _overflowing(torch, m):
    with pytest.raises(mg.FemGpuError) as e:
        _assemble(torch, m, None)
    assert e.value.status == 3  # FEM_GPU_NONFINITE


@pytest.mark.gpu
@pytest.mark.parametrize("at", [0, 537, -1])
@pytest.mark.parametrize("kind", ["E", "rho", "distorted"])
@pytest.mark.parametrize("p", [1, 2])
def test_one_overflowing_solid_cell_is_reported(torch, p, kind, at):
    """One modulus of 1e308 among ordinary ones: every kernel that stores values reports
    the block, as the element loop does."""
    ne = (10, 10, 11)
    mesh = mg.hmr_uniform_mesh(3, ne, (1e-3, 1.0, 1.0), p)
    if kind == "distorted":
        mesh = distort(mesh, 3, ne, 1e-5, 9)
    nc = len(mesh["cells"])
    E = np.ones(nc)
    E[at] = 1e308
    for pin in (False, True):
        m = mg.FemModel(3, mesh, mg.SHAPE_GENERAL if kind == "distorted" else mg.SHAPE_RECTANGULAR)
        m.add_bulk_set(np.arange(nc, dtype=np.int32), E, 0.49, mg.RULE_HEX_2x2x2, mg.MODEL_3D,
                       node_density=np.ones(len(mesh["coords"])) if kind == "rho" else None)
        m.finalize()
        if pin:
            m.set_variant(0, 2)
        before = m.launch_count()
        _overflowing(torch, m)
        if not pin and (p == 2 or kind == "rho"):
            assert m.launch_count() - before > 1


@pytest.mark.gpu
@pytest.mark.parametrize("at", [0, 17, -1])
@pytest.mark.parametrize("p", [1, 2, 3])
def test_one_overflowing_plane_cell_or_facet_is_reported(torch, p, at):
    ne = (9, 6)
    mesh = mg.hmr_uniform_mesh(2, ne, (1e-3, 1.0), p)
    nc = len(mesh["cells"])
    E = np.ones(nc)
    E[at] = 1e308
    left = np.arange(0, nc, ne[0], dtype=np.int32)
    for side in (False, True):
        m = mg.FemModel(2, mesh, mg.SHAPE_RECTANGULAR)
        m.add_bulk_set(np.arange(nc, dtype=np.int32), np.ones(nc) if side else E, 0.49, mg.RULE_QUAD_2x2,
                       mg.MODEL_PLANE_STRAIN)
        Es = np.ones(len(left))
        if side:
            Es[at % len(left)] = 1e308
        m.add_side_set(mg.IWG_STRUC_LINEAR_DIRICHLET_SYMMETRIC_NITSCHE, left, np.full(len(left), 3), Es, 0.49,
                       mg.RULE_BAR_3, mg.MODEL_PLANE_STRAIN, alpha=100.0)
        m.finalize()
        _overflowing(torch, m)


@pytest.mark.gpu
def test_mirrored_quadratic_cells_assemble_to_zero(torch):
    """Points of negative volume are skipped, also where the cells go through the stencil."""
    ne = (10, 10, 11)
    mesh = distort(mg.hmr_uniform_mesh(3, ne, [1.0] * 3, 2), 3, ne, 0.2, 9)
    mesh["coords"] = mesh["coords"] * np.array([-1.0, 1.0, 1.0])
    nc = len(mesh["cells"])
    m = mg.FemModel(3, mesh, mg.SHAPE_GENERAL)
    m.add_bulk_set(np.arange(nc, dtype=np.int32), uniform01(3, nc) + 0.1, 0.3, mg.RULE_HEX_2x2x2, mg.MODEL_3D)
    m.finalize()
    u = torch.tensor(uniform01(5, m.num_adofs) - 0.5, device="cuda")
    vals, rhs = _assemble(torch, m, u)
    y = torch.full_like(u, float("nan"))
    m.apply(u, y)
    torch.cuda.synchronize()
    assert not vals.any() and not rhs.any() and not y.any()
