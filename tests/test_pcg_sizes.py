"""Jacobi-PCG on both sides of the sizes up to which one cluster solves (5,120 rows,
and rows that fit its shared memory) and an iteration is two launches (one row per lane
group, one product block per SM: 9,728 rows with 152 SMs), against the allocation-free
entry point, whose iteration is four launches."""
import pytest
import scipy.sparse as sp

import moris_gb300 as mg
from tests.common import problem, rel_err

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    t = pytest.importorskip("torch")
    if not t.cuda.is_available():
        pytest.skip("no CUDA device")
    return t


def _system(torch, dim, ne):
    prod, _, _ = problem(dim, ne, 1, sides=True)
    prod.set_stream(torch.cuda.current_stream().cuda_stream)
    prod.finalize()
    rp, ci = prod.graph()
    vals = torch.empty(prod.nnz, dtype=torch.float64, device="cuda")
    rhs = torch.empty(prod.num_adofs, dtype=torch.float64, device="cuda")
    prod.assemble(None, vals, rhs)
    return prod, torch.tensor(rp, device="cuda"), torch.tensor(ci, device="cuda"), vals, -rhs


@pytest.mark.parametrize("dim,ne", [(2, (2, 2)), (2, (39, 63)), (2, (39, 64)), (2, (63, 75)), (2, (63, 76)), (3, (4, 3, 5)), (3, (13, 14, 14))])
def test_pcg_matches_noalloc(torch, dim, ne):
    """Solutions to the 1e-8 of the solver tests, iteration counts as there; no
    iteration from the solution; at a limit of 37, no multiple of the 32 captured
    iterations, the 37th iterate and not a neighbour of it (a bound on their distance
    from one another would be a bound on how CG amplifies the rounding of its sums)."""
    prod, rp, ci, vals, b = _system(torch, dim, ne)
    x, y = torch.zeros_like(b), torch.zeros_like(b)
    rx = prod.pcg(rp, ci, vals, b, x, rel_tol=1e-10)
    ry = prod.pcg_noalloc(rp, ci, vals, b, y, rel_tol=1e-10)
    torch.cuda.synchronize()
    assert rx["converged"] and rx["rel_residual"] <= 1e-10
    assert abs(rx["iterations"] - ry["iterations"]) <= max(3, ry["iterations"] // 20)
    assert rel_err(x.cpu().numpy(), y.cpu().numpy()) <= 1e-8
    again = prod.pcg(rp, ci, vals, b, x, rel_tol=1e-6)
    assert again["converged"] and again["iterations"] == 0
    if rx["iterations"] > 45:
        steps = {}
        for n in (36, 37, 38):
            steps[n] = torch.zeros_like(b)
            with pytest.raises(mg.FemGpuError) as ei:
                prod.pcg_noalloc(rp, ci, vals, b, steps[n], rel_tol=1e-14, max_iter=n)
            assert ei.value.status == 10  # NOT_CONVERGED
        x.zero_()
        with pytest.raises(mg.FemGpuError) as ei:
            prod.pcg(rp, ci, vals, b, x, rel_tol=1e-14, max_iter=37)
        assert ei.value.status == 10
        torch.cuda.synchronize()
        off = {n: float(torch.linalg.norm(x - y)) for n, y in steps.items()}
        assert off[37] < 1e-3 * min(off[36], off[38]), off


def test_rows_longer_than_the_models_graph(torch):
    """A matrix of the model's size with longer rows (the square of the operator plus a
    shift) leaves the cluster, which is laid out for the model's rows."""
    prod, rp, ci, vals, b = _system(torch, 2, (12, 9))
    n = prod.num_adofs
    A = sp.csr_matrix((vals.cpu().numpy(), ci.cpu().numpy(), rp.cpu().numpy()), shape=(n, n))
    A = (A + A.T) * 0.5
    B = (A @ A + abs(A).max() ** 2 * sp.identity(n)).tocsr()
    B.sort_indices()
    assert (B.indptr[1:] - B.indptr[:-1]).max() > 18
    rp, ci = torch.tensor(B.indptr, dtype=torch.int32, device="cuda"), torch.tensor(B.indices, dtype=torch.int32,
                                                                                    device="cuda")
    vals = torch.tensor(B.data, device="cuda")
    x, y = torch.zeros_like(b), torch.zeros_like(b)
    rx = prod.pcg(rp, ci, vals, b, x, rel_tol=1e-10)
    ry = prod.pcg_noalloc(rp, ci, vals, b, y, rel_tol=1e-10)
    torch.cuda.synchronize()
    assert rx["converged"] and abs(rx["iterations"] - ry["iterations"]) <= max(3, ry["iterations"] // 20)
    assert rel_err(x.cpu().numpy(), y.cpu().numpy()) <= 1e-8
