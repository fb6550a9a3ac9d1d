"""The one-launch ADMM loop with the masked transform (a disc of pixels and the
coefficients that reach it), at every number of levels it takes, against the
level-by-level kernels, inside the reconstruction loop that sets the masks.

Tolerance: the two run the same FP32 arithmetic and differ in the order of the
FP64 sums that decide when to stop, so three outer steps agree to 1e-5 (1e-6 per
map, as without masks)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import imgrecsrc_b200 as ct  # noqa: E402
from imgrecsrc_b200 import bhc, phantom  # noqa: E402
from oracle import wavelet_oracle as W  # noqa: E402


@pytest.mark.parametrize("L", [2, 3, 4, 5, 6])
def test_masked_levels(L, monkeypatch):
    n, J = 128, 8
    g = ct.Geometry(n, 180, 72, 72, 1.0, 1.0, 600.0)
    pr = ct.Projector(g)
    model = bhc.BHCModel(pr, bhc.kappa_nodes(J), 2.0 / n)
    truth = torch.from_numpy(phantom.two_material_phantom(n, seed=2).astype(np.float32)).cuda()
    m = torch.exp(-0.5 * 2.0 / n * pr.forward(truth))
    yy, xx = np.mgrid[0:n, 0:n]
    mask = torch.from_numpy((xx - 61.0) ** 2 + (yy - 66.0) ** 2 < 50.0 ** 2).cuda()

    def run():
        x = torch.full((n, n), 1.0, device="cuda")
        Ie = torch.full((J,), 1.0 / J, device="cuda", dtype=torch.float64)
        st = model.reconstruct(x, Ie, m, iterations=3, x_step=1e-3, method="npg", proximal="wvltADMM", u=1e-2,
                               wvlt_filter=W.daubcqf(2), wvlt_levels=L, mask=mask)
        return x, st["inner_iterations"]

    x, inner = run()
    monkeypatch.setenv("CTPRJ_WVLT_KERNEL", "levels")
    ref, inner_ref = run()
    assert inner == inner_ref > 0
    assert not x[~mask].any() and x[mask].any()
    assert ((x - ref).norm() / ref.norm()).item() < 1e-5
