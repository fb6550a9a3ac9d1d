"""The staged backprojection (k_backward_tiled) at the sizes where it can go
wrong, against the FP64 oracle: one pixel past and one short of a tile and of a
warp's square, images smaller than a square, detectors that end inside the
image, views split over one to eight blocks, windows from two detectors to the
general loop, beams narrower and wider than the pitch, views that stop short of
the turn, and the batched launch's sequential parts.

Tolerance: a weight is off by at most a few units of 1e-7 (FP32 arithmetic on
operands of at most a few pixels) and the sums add FP32 rounding over at most
a few hundred terms: 1e-5 relative L2 holds both with a margin, the bound of
the projector tests.  A beam wider than the pitch keeps the bound of
test_beam_wider_than_the_pitch (1e-4): there a shadow edge's rounding decides
weights that are not near zero."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import imgrecsrc_b200 as ct  # noqa: E402
import oracle  # noqa: E402
from imgrecsrc_b200 import batch  # noqa: E402

# (n, W, np, prjFull, dSize, effectiveRate, d)
CASES = [(1, 3, 4, 4, 1, 1, 0), (3, 5, 8, 8, 1, 1, 30), (15, 23, 12, 24, 1, 1, 0), (16, 24, 20, 20, 1, 1, 64),
         (17, 25, 32, 32, 1, 1, 50), (31, 45, 33, 36, 1, 1, 93), (33, 46, 20, 40, 1, 1, 0), (34, 20, 40, 40, 1, 1, 120),
         (63, 91, 64, 128, 1, 1, 0), (65, 60, 30, 100, 1, 1, 400), (97, 139, 128, 128, 1, 1, 200),
         (129, 184, 260, 260, 1, 1, 320), (255, 300, 64, 128, 1, 1, 0), (48, 40, 96, 96, 2.5, 1, 100),
         (48, 140, 96, 96, 0.5, 1, 150), (64, 200, 44, 88, 0.45, 1, 0), (64, 91, 60, 120, 1, 0.6, 0),
         (64, 91, 60, 60, 1, 0.6, 160), (64, 91, 48, 48, 1, 1.3, 160), (64, 91, 48, 96, 1, 1.3, 0),
         (40, 120, 36, 36, 1, 1, 62)]


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("case", CASES, ids=str)
def test_tiles_against_the_oracle(case):
    g = ct.Geometry(*case)
    y = np.random.default_rng(g.n).standard_normal((g.np, g.prjWidth)).astype(np.float32)
    dy = torch.from_numpy(y).cuda()
    pr = ct.Projector(g)
    b = pr.backward(dy)
    tol = 1e-4 if g.effectiveRate > 1 else 1e-5
    assert rel(b.double().cpu().numpy(), oracle.backward(g, y.astype(np.float64))) < tol
    assert rel(pr.fbp(dy).double().cpu().numpy(), oracle.fbp(g, y.astype(np.float64))) < 1e-4
    # the same bits again, and from one block that takes the parts in turn
    out = torch.full((g.n, g.n), float("nan"), device="cuda")
    bt = batch.Batch([g])
    bt.bind(bsinos=[dy], bimgs=[out])
    bt.backward()
    assert torch.equal(pr.backward(dy), b) and torch.equal(out, b)


def test_a_bad_sample_stays_on_its_ray():
    """An infinite sample reaches the pixels its beam meets and at most the
    next window's width beyond (weights of zero), no further."""
    g = ct.Geometry(64, 91, 64, 128, 1, 1, 0)
    y = torch.zeros(g.np, g.prjWidth, device="cuda")
    y[0, 50] = float("inf")            # view 0: t = 50 - 45 = 5 meets the column x = 5
    b = ct.Projector(g).backward(y)
    cols = torch.nonzero(~torch.isfinite(b).all(0)).squeeze(1).cpu().numpy() - 32
    assert 5 in cols and np.abs(cols - 5).max() <= 3
