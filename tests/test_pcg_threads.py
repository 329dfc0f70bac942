"""Small systems of different sizes solved by several threads at once, a context each: the
one-cluster solver's launch must not depend on what another thread's solve has set up."""
import threading

import pytest

import moris_gb300 as mg
from tests.common import problem, rel_err

pytestmark = pytest.mark.gpu


def test_solves_of_different_sizes_side_by_side():
    """One thread solves 5,120 rows (104 KB of shared memory per CTA, the most the solver
    asks for), four threads solve 18 rows in a loop meanwhile.  Every solve succeeds with
    the solution it has alone (to the 1e-8 of the solver tests)."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")

    def system(ne):
        m, _, _ = problem(2, ne, 1, sides=True)
        s = torch.cuda.Stream()
        m.set_stream(s.cuda_stream)
        m.finalize()
        rp, ci = m.graph()
        vals = torch.empty(m.nnz, dtype=torch.float64, device="cuda")
        rhs = torch.empty(m.num_adofs, dtype=torch.float64, device="cuda")
        m.assemble(None, vals, rhs)
        rp, ci, b = torch.tensor(rp, device="cuda"), torch.tensor(ci, device="cuda"), -rhs
        torch.cuda.synchronize()
        return m, s, rp, ci, vals, b

    def solve(a, x):
        m, _, rp, ci, vals, b = a
        return m.pcg(rp, ci, vals, b, x, rel_tol=1e-10)

    large, small = system((39, 63)), [system((2, 2)) for _ in range(4)]
    assert large[0].num_adofs == 5120 and small[0][0].num_adofs == 18
    ref = torch.zeros_like(large[5])
    solve(large, ref)
    out = [torch.zeros_like(ref) for _ in range(20)]
    xs = [torch.zeros_like(a[5]) for a in small]
    torch.cuda.synchronize()
    stop, errors, solved = threading.Event(), [], [0] * len(small)

    def loop(k):
        try:
            while not stop.is_set():
                solve(small[k], xs[k])  # from the second call on the solution itself: no iteration
                solved[k] += 1
        except mg.FemGpuError as e:
            errors.append(e)

    threads = [threading.Thread(target=loop, args=(k,)) for k in range(len(small))]
    for t in threads:
        t.start()
    try:
        for x in out:
            solve(large, x)
    finally:
        stop.set()
        for t in threads:
            t.join()
    torch.cuda.synchronize()
    assert not errors and min(solved) > 0
    for x in out:
        assert rel_err(x.cpu().numpy(), ref.cpu().numpy()) <= 1e-8
