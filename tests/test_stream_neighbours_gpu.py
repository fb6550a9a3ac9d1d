"""Streaming backprojection of slices that lie one behind the other in memory, at
boundaries that are no multiple of a cache sector, each copied and published while
the kernel runs: a slice's first samples must not come from a cache line that was
read with its neighbour's last ones.  Equal to the plain backprojection."""
import threading
import time

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import imgrecsrc_b200 as ct  # noqa: E402
from imgrecsrc_b200 import batch  # noqa: E402


# (at a detector pitch of 0.2 a tile's shadow is too wide to be staged)
@pytest.mark.parametrize("pitch, d", [(1.0, 0.0), (1.0, 300.0), (0.2, 0.0)], ids=["parallel", "fan", "unstaged"])
def test_slices_side_by_side(pitch, d):
    g = ct.Geometry(60, 85, 37, 40, pitch, 1.0, d)
    count, size = 16, 37 * 85   # 3145 samples: one past a multiple of eight
    gen = torch.Generator().manual_seed(6)
    host = torch.randn(count, size, generator=gen).pin_memory()
    packed = torch.full((count * size,), float("nan"), device="cuda")
    sinos = [packed[i * size:(i + 1) * size] for i in range(count)]
    pr = ct.Projector(g)
    refs = [pr.backward(h.cuda().view(g.np, g.prjWidth)) for h in host]
    outs = [torch.empty(g.n, g.n, device="cuda") for _ in range(count)]
    b = batch.Batch([g] * count)
    b.bind(None, None, sinos, outs)
    copies, side = torch.cuda.Stream(), torch.cuda.Stream()   # neither waits for the default stream
    for _ in range(3):
        packed.fill_(float("nan"))
        flags = batch.StreamFlags(count)
        torch.cuda.synchronize()

        def publish():
            for i in range(count):
                with torch.cuda.stream(copies):
                    sinos[i].copy_(host[i], non_blocking=True)
                copies.synchronize()
                flags.publish(i)
                time.sleep(0.002)
        th = threading.Thread(target=publish)
        th.start()
        code, status = batch.stream_backward(b, flags, 5.0, stream=side)
        th.join()
        torch.cuda.synchronize()
        assert code == ct._lib.CTPRJ_OK and status == [0] * count
        for o, r in zip(outs, refs):
            assert torch.equal(o, r)
        flags.close()
