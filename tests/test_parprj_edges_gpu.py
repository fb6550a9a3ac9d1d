"""The edge form of the FP64 parallel operator (unit beams) beside the
pixel-by-pixel form: axis-aligned and diagonal angles and their neighbours,
images smaller than a warp's detectors, detectors fewer and more than the image
is wide, sparse masks, sums shared by several warps and not, other beam widths,
and a value that is not finite.

Tolerance 1e-12 relative L2, as the operator's other tests: both sides are FP64
and differ in rounding only."""
import numpy as np
import pytest

import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from imgrecsrc_b200 import mex  # noqa: E402

ANGLES = [0, 1e-9, 0.4, 1, 44, 44.5, 45, 45.3, 46, 89, 89.6, 90, 90.2, 134.7, 135, 179.5, 180, 270, -30, -45, 315, 359.9]


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a) - b) / max(np.linalg.norm(b), 1e-300))


@pytest.mark.parametrize("bw", [1.0, 0.7, 1.6])
@pytest.mark.parametrize("nc,nr,W,fill", [(1, 1, 3, 1.0), (5, 9, 7, 1.0), (31, 20, 31, 0.5), (32, 33, 70, 0.1), (64, 64, 91, 0.8),
                                          (100, 63, 40, 1.0)])
def test_against_the_oracle(nc, nr, W, fill, bw):
    rng = np.random.default_rng(nc)
    mask = np.flatnonzero(rng.uniform(size=nc * nr) < fill).astype(np.float64)
    x, y = rng.standard_normal(mask.size), rng.standard_normal(len(ANGLES) * W)
    conf = dict(bw=bw, nc=nc, nr=nr, np=len(ANGLES), prjWidth=W, theta=np.array(ANGLES, np.float64))
    fx, by = mex.mParPrj(x, mask, conf, "forward"), mex.mParPrj(y, mask, conf, "backward")
    assert rel(fx, np.asarray(oracle.par_forward(x, mask, conf)).ravel()) < 1e-12
    assert rel(by, np.asarray(oracle.par_backward(y, mask, conf)).ravel()) < 1e-12


@pytest.mark.parametrize("angles", [40, 400])
def test_shared_and_whole_sums(angles):
    n, W = 150, 213
    rng = np.random.default_rng(angles)
    mask = np.arange(n * n, dtype=np.float64)
    conf = dict(bw=1.0, nc=n, nr=n, np=angles, prjWidth=W, theta=np.arange(angles) * 180.0 / angles)
    x, y = rng.uniform(size=mask.size), rng.standard_normal(angles * W)
    fx, by = mex.mParPrj(x, mask, conf, "forward"), mex.mParPrj(y, mask, conf, "backward")
    assert rel(fx, np.asarray(oracle.par_forward(x, mask, conf)).ravel()) < 1e-12
    assert rel(by, np.asarray(oracle.par_backward(y, mask, conf)).ravel()) < 1e-12
    assert np.array_equal(fx, mex.mParPrj(x, mask, conf, "forward"))
    assert np.array_equal(by, mex.mParPrj(y, mask, conf, "backward"))


def test_an_infinite_pixel_reaches_its_detectors_only():
    n, W = 40, 57
    mask = np.arange(n * n, dtype=np.float64)
    conf = dict(bw=1.0, nc=n, nr=n, np=len(ANGLES), prjWidth=W, theta=np.array(ANGLES, np.float64))
    x = np.ones(n * n)
    x[17 * n + 23] = np.inf
    assert np.array_equal(np.isposinf(mex.mParPrj(x, mask, conf, "forward")),
                          np.isposinf(np.asarray(oracle.par_forward(x, mask, conf)).ravel()))
