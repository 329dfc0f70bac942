"""Matrix-free products of one lattice model on several streams and in a captured graph:
the model's workspaces must not be shared by work that may run at the same time."""
import pytest

import moris_gb300 as mg
from tests.common import RTOL, problem, rel_err, uniform01

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    t = pytest.importorskip("torch")
    if not t.cuda.is_available():
        pytest.skip("no CUDA device")
    return t


@pytest.mark.parametrize("shape,density", [(mg.SHAPE_RECTANGULAR, False), (mg.SHAPE_RECTANGULAR, True),
                                           (mg.SHAPE_GENERAL, False)], ids=["bricks", "density", "distorted"])
def test_products_on_two_streams_and_in_a_graph(torch, shape, density):
    m, _, _ = problem(3, (17, 16, 15), 2, shape, mg.RULE_HEX_2x2x2, density=density)
    m.finalize()
    m.set_stream(torch.cuda.current_stream().cuda_stream)
    x = [torch.tensor(uniform01(s, m.num_adofs) - 0.5, device="cuda") for s in (5, 6)]
    ref = [torch.empty_like(v) for v in x]
    for v, r in zip(x, ref):
        m.apply(v, r)
    torch.cuda.synchronize()
    y = [[torch.full_like(x[0], float("nan")) for _ in range(8)] for _ in x]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    for k in range(8):
        for s, v, out in zip(streams, x, y):
            m.set_stream(s.cuda_stream)
            m.apply(v, out[k])
    torch.cuda.synchronize()
    for r, out in zip(ref, y):
        for o in out:
            assert rel_err(o.cpu().numpy(), r.cpu().numpy()) <= RTOL
    # a captured product replayed beside direct ones
    g, yg = torch.cuda.CUDAGraph(), torch.full_like(x[0], float("nan"))
    with torch.cuda.graph(g, stream=streams[0]):
        m.set_stream(torch.cuda.current_stream().cuda_stream)
        m.apply(x[0], yg)
    m.set_stream(streams[1].cuda_stream)
    torch.cuda.synchronize()
    for k in range(8):
        with torch.cuda.stream(streams[0]):
            g.replay()
        m.apply(x[1], y[1][k])
    torch.cuda.synchronize()
    assert rel_err(yg.cpu().numpy(), ref[0].cpu().numpy()) <= RTOL
    for o in y[1]:
        assert rel_err(o.cpu().numpy(), ref[1].cpu().numpy()) <= RTOL
