"""Matrix-free products of one lattice model from two threads in turn, each on its
per-thread default stream.  Both streams have the same handle, so the model's workspaces
cannot be ordered by comparing handles.  A thread ends only when its stream has run."""
import threading

import pytest

import moris_gb300 as mg
from tests.common import RTOL, problem, rel_err, uniform01

pytestmark = pytest.mark.gpu

PER_THREAD_STREAM = 2  # cudaStreamPerThread


@pytest.mark.parametrize("shape,density", [(mg.SHAPE_RECTANGULAR, False), (mg.SHAPE_RECTANGULAR, True),
                                           (mg.SHAPE_GENERAL, False)], ids=["bricks", "density", "distorted"])
def test_products_on_the_per_thread_streams_of_two_threads(shape, density):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    m, _, _ = problem(3, (17, 16, 15), 2, shape, mg.RULE_HEX_2x2x2, density=density)
    m.finalize()
    x = [torch.tensor(uniform01(s, m.num_adofs) - 0.5, device="cuda") for s in (5, 6)]
    ref = [torch.empty_like(v) for v in x]
    for v, r in zip(x, ref):
        m.apply(v, r)
    rounds = 8
    y = [[torch.full_like(x[0], float("nan")) for _ in range(rounds)] for _ in x]
    torch.cuda.synchronize()
    m.set_stream(PER_THREAD_STREAM)
    turn, errors = [threading.Semaphore(1), threading.Semaphore(0)], []

    def products(k):
        for i in range(rounds):
            turn[k].acquire()
            try:
                m.apply(x[k], y[k][i])  # returns before it has run
            except mg.FemGpuError as e:
                errors.append(e)
            finally:
                turn[1 - k].release()
        torch.cuda.ExternalStream(PER_THREAD_STREAM).synchronize()

    threads = [threading.Thread(target=products, args=(k,)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors
    for r, out in zip(ref, y):
        for o in out:
            assert rel_err(o.cpu().numpy(), r.cpu().numpy()) <= RTOL
