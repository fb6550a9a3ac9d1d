"""The forward projection into the image's own memory: the pass reads the image
once, into the quad image, and writes the sinogram (the zero column of an even
width among it) only when that is done.  Equal to the pass into a buffer of its
own, bit for bit, since the sums are the same."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import imgrecsrc_b200 as ct  # noqa: E402


@pytest.mark.parametrize("g", [ct.Geometry(64, 90, 48, 48, 1.0, 1.0, 200.0), ct.Geometry(257, 366, 180, 360, 1.0, 1.0, 0.0),
                               ct.Geometry(1024, 1454, 720, 720, 1.0, 1.0, 4096.0)], ids=lambda g: str(g.n))
def test_sinogram_on_the_image(g):
    x = torch.rand(g.n, g.n, device="cuda", generator=torch.Generator(device="cuda").manual_seed(2))
    pr = ct.Projector(g)
    ref = pr.forward(x)
    buf = torch.empty(max(x.numel(), ref.numel()), device="cuda")
    for _ in range(5):
        buf[:x.numel()] = x.reshape(-1)
        s = pr.forward(buf[:x.numel()].view(g.n, g.n), out=buf[:ref.numel()].view(g.np, g.prjWidth))
        assert torch.equal(s, ref)
