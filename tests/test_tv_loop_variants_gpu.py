"""The one-launch TV loop's variants (32-row tiles at up to two blocks per SM,
64-row tiles beyond, 32-row tiles at up to four per SM where the 64-row ones do
not fit), one ragged size each, against the FP64 restatement.

Tolerance: FP32 arithmetic of some 30 iterations of a contraction, each rounding
at 6e-8 of its terms: 1e-4 relative L2, as for the other sizes of this kernel."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from imgrecsrc_b200 import tv  # noqa: E402
from oracle import tv_oracle as TVO  # noqa: E402


@pytest.mark.parametrize("kind", ["iso", "l1"])
@pytest.mark.parametrize("shape", [(590, 1025), (1009, 701), (32, 20481), (33, 12803)])
def test_variants(shape, kind):
    X = np.random.default_rng(3).standard_normal(shape).astype(np.float32) + 0.5
    d = torch.from_numpy(X).cuda()
    out, it = tv.denoise(d, 0.2, 0.0, 30, tv_type=kind, n_row=shape[1], n_col=shape[0])
    ref, ito = TVO.tv_denoise(X.astype(np.float64), 0.2, tv=kind, max_iter=30, eps=0.0)
    assert it == ito == 30
    assert np.linalg.norm(out.double().cpu().numpy() - ref) < 1e-4 * np.linalg.norm(ref)
    again, _ = tv.denoise(d, 0.2, 0.0, 30, tv_type=kind, n_row=shape[1], n_col=shape[0])
    assert torch.equal(out, again)
