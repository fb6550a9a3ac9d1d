"""The fused two-tap ADMM iteration at few levels on images of many tiles: a
2^L x 2^L tile writes its own partial sums, so few levels need room for many
more of them than the level passes have blocks.

Tolerance: as the fixed-iteration tests of test_wavelet_gpu.py (1e-4 relative
L2 against the FP64 restatement after tens of iterations in FP32)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from imgrecsrc_b200 import wavelet  # noqa: E402
from oracle import wavelet_oracle as W  # noqa: E402


@pytest.mark.parametrize("L,shape", [(1, (128, 256)), (2, (256, 320)), (3, (384, 320)), (4, (640, 704)), (5, (640, 704))])
def test_many_tiles_of_few_levels(L, shape):
    rng = np.random.default_rng(L)
    a = (rng.standard_normal(shape) + 0.3).astype(np.float32)
    h = W.daubcqf(2)
    al, it = wavelet.admm(torch.from_numpy(a).cuda(), 0.4, h, L, relative_tol=0.0, max_itr=25)
    alo, ito = W.admm(a.astype(np.float64), 0.4, h, L, rel_tol=0.0, max_itr=25)
    assert it == ito == 26
    assert np.linalg.norm(al.double().cpu().numpy() - alo) / np.linalg.norm(alo) < 1e-4
