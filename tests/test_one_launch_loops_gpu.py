"""The proximal maps whose whole iteration loop is one cooperative launch
(k_tv_loop, k_admm_loop), at the edges of their tiles and of the sizes they
take, against the FP64 restatements and the launch-per-iteration kernels.

Tolerance: the maps run the same FP32 arithmetic as the launch-per-iteration
kernels, whose tests hold 1e-4 relative L2 against FP64 after tens of
iterations; the two paths differ only in the order of FP64 sums that decide
when to stop, so a fixed number of iterations agrees to 1e-6."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from imgrecsrc_b200 import tv, wavelet  # noqa: E402
from oracle import tv_oracle as TVO  # noqa: E402
from oracle import wavelet_oracle as W  # noqa: E402


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("kind", ["iso", "l1"])
@pytest.mark.parametrize("shape", [(2, 2), (2, 150), (150, 2), (31, 63), (32, 64), (33, 65), (64, 128), (97, 130)])
def test_tv_tile_edges(shape, kind):
    X = np.random.default_rng(shape[0] + shape[1]).standard_normal(shape).astype(np.float32) + 0.5
    d = torch.from_numpy(X).cuda()
    out, it = tv.denoise(d, 0.2, 0.0, 45, tv_type=kind, n_row=shape[1], n_col=shape[0])
    ref, ito = TVO.tv_denoise(X.astype(np.float64), 0.2, tv=kind, max_iter=45, eps=0.0)
    assert it == ito == 45
    assert rel(out.double().cpu().numpy(), ref) < 1e-4
    # the stopping rule, decided by every block for itself
    out, it = tv.denoise(d, 0.2, 1e-3, 400, tv_type=kind, n_row=shape[1], n_col=shape[0])
    ref, ito = TVO.tv_denoise(X.astype(np.float64), 0.2, tv=kind, max_iter=400, eps=1e-3)
    assert abs(it - ito) <= 2
    z, it = tv.denoise(d, 0.2, 0.0, 0, tv_type=kind, n_row=shape[1], n_col=shape[0])
    assert it == 0 and not z.any()


@pytest.mark.parametrize("n", [1056, 1216, 1504])
def test_tv_on_both_sides_of_the_size_limit(n):
    """The largest images of the one-launch loop and the first of the
    launch-per-iteration kernel give the same map: the centre of an image
    whose border repeats far from it does not depend on the size."""
    x = torch.zeros(n, n, device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(1)
    x[300:500, 300:500] = torch.rand(200, 200, device="cuda", generator=gen)
    out, it = tv.denoise(x, 0.1, 0.0, 30)
    small = x[200:600, 200:600].contiguous()
    ref, its = tv.denoise(small, 0.1, 0.0, 30)
    assert it == its == 30
    a, b = out[300:500, 300:500], ref[100:300, 100:300]
    assert ((a - b).norm() / b.norm()).item() < 1e-5


@pytest.mark.parametrize("L", [2, 3, 4, 5, 6])
@pytest.mark.parametrize("shape", [(64, 64), (64, 192), (128, 64), (192, 320)])
def test_admm_tiles(L, shape, monkeypatch):
    rng = np.random.default_rng(L)
    a = torch.from_numpy((rng.standard_normal(shape) + 0.3).astype(np.float32)).cuda()
    init = torch.from_numpy(np.maximum(rng.standard_normal(shape), 0).astype(np.float32)).cuda()
    h = W.daubcqf(2)
    for tol, iters, start in ((0.0, 45, init), (1e-4, 300, None)):
        al, it = wavelet.admm(a, 0.4, h, L, relative_tol=tol, max_itr=iters, init=start)
        monkeypatch.setenv("CTPRJ_WVLT_KERNEL", "levels")
        ref, itr = wavelet.admm(a, 0.4, h, L, relative_tol=tol, max_itr=iters, init=start)
        monkeypatch.delenv("CTPRJ_WVLT_KERNEL")
        assert it == itr
        assert ((al - ref).norm() / ref.norm()).item() < 1e-6
    z, it = wavelet.admm(torch.zeros_like(a), 0.4, h, L)
    assert it == 0 and not z.any()
