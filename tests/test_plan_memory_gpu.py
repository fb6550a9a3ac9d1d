"""Plans share the device's memory pool: a plan whose memory was another's gives
its own results, and a plan may be destroyed while its passes still run."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import imgrecsrc_b200 as ct  # noqa: E402

GEOMS = [ct.Geometry(64, 90, 48, 48, 1.0, 1.0, 200.0), ct.Geometry(256, 363, 180, 360, 1.0, 1.0, 0.0),
         ct.Geometry(257, 300, 120, 120, 1.0, 1.0, 900.0), ct.Geometry(512, 729, 360, 360, 1.0, 1.0, 2048.0)]


def _pair(pr, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.rand(pr.img_shape, device="cuda", generator=gen)
    s = pr.forward(x)
    return s, pr.backward(s)


def test_plans_kept_and_destroyed_in_any_order():
    first = []
    for i, g in enumerate(GEOMS):
        pr = ct.Projector(g)
        first.append(_pair(pr, i))
        torch.cuda.synchronize()
        pr.close()
    plans = [ct.Projector(GEOMS[i % 4]) for i in range(12)]
    for i in (5, 0, 7, 2, 9):
        plans[i].close()
        plans[i] = ct.Projector(GEOMS[i % 4])
    for i, pr in enumerate(plans):
        assert all(torch.equal(a, b) for a, b in zip(_pair(pr, i % 4), first[i % 4]))


def test_a_plan_destroyed_while_its_passes_run():
    pr = ct.Projector(GEOMS[3])
    want = _pair(pr, 3)
    stream = torch.cuda.Stream()
    for _ in range(3):
        torch.cuda.synchronize()
        x = torch.rand(pr.img_shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(3))
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            for _ in range(20):
                s = pr.forward(x)
                b = pr.backward(s)
        pr.close()
        assert stream.query()          # destroying waited for the passes
        other = [ct.Projector(GEOMS[i]) for i in (3, 1)]   # into the same memory
        for o, i in zip(other, (3, 1)):
            _pair(o, i)
        torch.cuda.synchronize()
        assert torch.equal(s, want[0]) and torch.equal(b, want[1])
        pr = other[0]
