"""The forward projection on fan geometries whose outer rays miss the image, some
of them nearly parallel to its columns (warps that have no rows at all): per
plan, batched and polychromatic, against the FP64 oracle.

Tolerance: FP32 sums of about a thousand terms whose weights are off by a few
units of 1e-7: 1e-5 relative L2, the bound of the projector tests."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import imgrecsrc_b200 as ct  # noqa: E402
import oracle  # noqa: E402
from imgrecsrc_b200 import batch, bhc  # noqa: E402

# (n, W, P, d), unit pitch and beam; the views of one eighth of the turn
GEOMS = [(1136, 1617, 668, 3408), (944, 1465, 716, 2360), (950, 1859, 504, 3800), (933, 2288, 672, 1866),
         (812, 2290, 940, 2436)]


@pytest.mark.parametrize("n, W, P, d", GEOMS)
def test_rays_beside_the_image(n, W, P, d):
    g = ct.Geometry(n, W, P // 8 + 1, P, 1.0, 1.0, float(d))
    x = np.random.default_rng(n).uniform(0, 1, (n, n)).astype(np.float32)
    dx = torch.from_numpy(x).cuda()
    pr = ct.Projector(g)
    s = pr.forward(dx)
    ref = oracle.forward(g, x.astype(np.float64))
    got = s.double().cpu().numpy()
    assert np.linalg.norm(got - ref) < 1e-5 * np.linalg.norm(ref)
    assert not got[ref == 0].any() and (ref == 0).any()   # the rays that miss
    out = torch.full((g.np, W), float("nan"), device="cuda")
    bt = batch.Batch([g])
    bt.bind(imgs=[dx], sinos=[out])
    bt.forward()
    assert torch.equal(out, s)
    # the polychromatic pass, on the same sums
    m = torch.rand(g.np, W, device="cuda", generator=torch.Generator(device="cuda").manual_seed(3))
    Ie = torch.full((7,), 1.0 / 7, dtype=torch.float64, device="cuda")
    model = bhc.BHCModel(pr, bhc.kappa_nodes(7), 1e-3)
    f, t = model.forward(dx, Ie, m).item(), model.terms(s, Ie, m).item()
    assert abs(f - t) <= 1e-12 * abs(t)
