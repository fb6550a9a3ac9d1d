"""The forward projection with its rows summed in parts (k_forward): images of
fewer rows than parts, rays that miss the image or part of it, the central
detector, views that stop short of the turn, and the batched launch, which sums
the parts one after the other; the polychromatic epilogue on the same sums.

Tolerance: FP32 sums of at most a few hundred terms whose weights are off by a
few units of 1e-7: 1e-5 relative L2, the bound of the projector tests."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import imgrecsrc_b200 as ct  # noqa: E402
import oracle  # noqa: E402
from imgrecsrc_b200 import batch, bhc  # noqa: E402

# (n, W, np, prjFull, dSize, effectiveRate, d)
CASES = [(1, 3, 4, 8, 1, 1, 0), (2, 4, 8, 8, 1, 1, 40), (5, 9, 7, 12, 1, 1, 20), (8, 40, 16, 32, 1, 1, 0),
         (15, 22, 24, 24, 1, 1, 64), (17, 70, 20, 40, 1, 1, 0), (33, 200, 36, 36, 1, 1, 100), (64, 30, 48, 96, 1, 1, 0),
         (97, 139, 33, 60, 1, 1, 300), (150, 140, 64, 128, 1, 1, 0), (96, 136, 72, 72, 0.5, 1, 200),
         (48, 68, 40, 40, 1, 0.6, 110), (48, 68, 40, 80, 1, 1.3, 0), (40, 60, 36, 36, 2.0, 1, 62)]


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("case", CASES, ids=str)
def test_parts_against_the_oracle(case):
    g = ct.Geometry(*case)
    x = np.random.default_rng(g.n).uniform(0, 1, (g.n, g.n)).astype(np.float32)
    dx = torch.from_numpy(x).cuda()
    pr = ct.Projector(g)
    s = pr.forward(dx)
    ref = oracle.forward(g, x.astype(np.float64))
    assert rel(s.double().cpu().numpy(), ref) < 1e-5
    out = torch.full((g.np, g.prjWidth), float("nan"), device="cuda")
    bt = batch.Batch([g])
    bt.bind(imgs=[dx], sinos=[out])
    bt.forward()
    assert torch.equal(pr.forward(dx), s) and torch.equal(out, s)


@pytest.mark.parametrize("case", [(33, 60, 36, 36, 1, 1, 100), (48, 66, 40, 80, 1, 1, 0)], ids=str)
def test_fused_likelihood_of_the_parts(case):
    """The fused forward evaluates every sinogram entry once: its f equals the
    unfused terms' on the same projections to the order of an FP64 sum."""
    g = ct.Geometry(*case)
    gen = torch.Generator(device="cuda").manual_seed(3)
    x = torch.rand(g.n, g.n, device="cuda", generator=gen) * 3
    m = torch.rand(g.np, g.prjWidth, device="cuda", generator=gen)
    Ie = torch.rand(7, dtype=torch.float64, device="cuda", generator=gen)
    pr = ct.Projector(g)
    model = bhc.BHCModel(pr, bhc.kappa_nodes(7), 0.05)
    f = model.forward(x, Ie, m).item()
    gx, gI = model.backward()
    t = model.terms(pr.forward(x), Ie, m).item()
    tx, tI = model.backward()
    assert abs(f - t) <= 1e-12 * abs(t)
    assert torch.equal(gx, tx) and torch.equal(gI, tI)
