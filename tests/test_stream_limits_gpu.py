"""The streaming backprojection's limit is for the host's publication: slices
published before the launch come out whatever the limit, also where it is shorter
than the work that a tile of the slice waits for (its sample rows)."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import imgrecsrc_b200 as ct  # noqa: E402
from imgrecsrc_b200 import batch  # noqa: E402


@pytest.mark.parametrize("limit", [1e-9, 1e-6, 1e-4])
def test_published_slices_are_never_late(limit):
    geoms = [ct.Geometry(256, 363, 360, 720, 1.0, 1.0, 0.0), ct.Geometry(96, 137, 60, 60, 1.0, 1.0, 400.0),
             ct.Geometry(200, 284, 400, 400, 1.0, 1.0, 900.0)]
    gen = torch.Generator(device="cuda").manual_seed(4)
    sinos = [torch.randn(g.np, g.prjWidth, device="cuda", generator=gen) for g in geoms]
    outs = [torch.full((g.n, g.n), float("nan"), device="cuda") for g in geoms]
    refs = [ct.Projector(g).backward(y) for g, y in zip(geoms, sinos)]
    b = batch.Batch(geoms)
    b.bind(None, None, sinos, outs)
    flags = batch.StreamFlags(len(geoms))
    for i in range(len(geoms)):
        flags.publish(i)
    torch.cuda.synchronize()
    for _ in range(5):
        for o in outs:
            o.fill_(float("nan"))
        code, status = batch.stream_backward(b, flags, limit)
        torch.cuda.synchronize()
        assert code == ct._lib.CTPRJ_OK and status == [0] * len(geoms)
        for o, r in zip(outs, refs):
            assert torch.equal(o, r)
    flags.close()
