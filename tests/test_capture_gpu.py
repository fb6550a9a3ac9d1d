"""The plan's passes in a captured CUDA graph: each is two launches of which the
second starts beside the first, and a replay follows the inputs as they are then.
Equal to the calls outside a graph, bit for bit, since the kernels are the same."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import imgrecsrc_b200 as ct  # noqa: E402
from imgrecsrc_b200 import bhc  # noqa: E402


@pytest.mark.parametrize("g", [ct.Geometry(64, 90, 48, 48, 1.0, 1.0, 200.0), ct.Geometry(256, 363, 180, 360, 1.0, 1.0, 0.0),
                               ct.Geometry(700, 1000, 360, 360, 1.0, 1.0, 2800.0)], ids=lambda g: str(g.n))
def test_replays_follow_the_inputs(g):
    gen = torch.Generator(device="cuda").manual_seed(7)
    pr = ct.Projector(g)
    model = bhc.BHCModel(pr, bhc.kappa_nodes(7), 0.01)
    Ie = torch.full((7,), 1.0 / 7, dtype=torch.float64, device="cuda")
    x = torch.rand(g.n, g.n, device="cuda", generator=gen)
    m = torch.rand(g.np, g.prjWidth, device="cuda", generator=gen)

    def step():
        s = pr.forward(x)
        b = pr.backward(s)
        f = model.forward(b * (1.0 / b.numel()), Ie, m)
        gx, gI = model.backward()
        return s, b, f, gx, gI
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = step()
    for _ in range(3):
        x.copy_(torch.rand(g.n, g.n, device="cuda", generator=gen))
        graph.replay()
        got = [t.clone() for t in out]
        ref = step()
        for a, b in zip(got, ref):
            assert torch.equal(a, b)
