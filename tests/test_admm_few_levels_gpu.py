"""The one-launch ADMM loop at two to four levels, where an iteration has no
barrier of the coarse levels, on images of one block per SM and of two: every
block goes by the same sums, so a run repeats bit for bit, and it follows the
level-by-level kernels.

Tolerance: the two run the same FP32 arithmetic and differ in the order of the
FP64 sums that set rho and stop: 1e-6 relative L2, as at the other sizes."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from imgrecsrc_b200 import wavelet  # noqa: E402
from oracle import wavelet_oracle as W  # noqa: E402


@pytest.mark.parametrize("L", [2, 3, 4])
@pytest.mark.parametrize("shape", [(64, 64), (768, 704), (1024, 1024)])
def test_blocks_agree(L, shape, monkeypatch):
    a = torch.from_numpy((np.random.default_rng(L).standard_normal(shape) + 0.3).astype(np.float32)).cuda()
    h = W.daubcqf(2)
    runs = [wavelet.admm(a, 0.4, h, L, relative_tol=1e-7, max_itr=120) for _ in range(10)]
    monkeypatch.setenv("CTPRJ_WVLT_KERNEL", "levels")
    ref, itr = wavelet.admm(a, 0.4, h, L, relative_tol=1e-7, max_itr=120)
    for al, it in runs:
        assert it == itr and torch.equal(al, runs[0][0])
    assert ((runs[0][0] - ref).norm() / ref.norm()).item() < 1e-6
