"""The staged backprojection's windows hold every detector that a pixel meets
(host-side check of the rule in square_view and pair_start, restated here; no
GPU).

A thread takes two pixels side by side; per view and 8 x 8 pixel square the rule
gives n detectors for each and the offset o of the window that starts later, and
the pair's first detector from the projection of its middle, held inside the
staged detectors.  A detector k meets the pixel at (u, v) along / across the
detector when |u - k G| < (G effectiveRate + |c - T s| + |s + T c|) / 2, with
G = dSize (d - v) / d and T = k dSize / d (parallel beam: G = dSize, T = 0); with
effectiveRate > 1 it also has to lie in the pixel's corner shadow
(prj/cpuPrj.c:81-105, :218-244).  Every detector that does is inside the window of
its pixel, for squares of random tiles and views."""
import numpy as np
import pytest

F = np.float32
PI_F = F(3.14159265359)
TILE, PAST = 16, 2
# (n, W, P, d, effectiveRate, dSize)
GEOMS = [(2048, 2048, 1440, 8192.0, 1.0, 1.0), (512, 1024, 360, 2048.0, 1.0, 1.0), (256, 363, 360, 0.0, 1.0, 1.0),
         (1024, 1024, 720, 2048.0, 1.0, 1.0), (128, 200, 180, 200.0, 1.0, 1.0), (64, 140, 60, 96.0, 1.0, 1.0),
         (64, 91, 60, 0.0, 0.5, 0.7), (97, 139, 120, 300.0, 0.8, 0.6), (48, 70, 40, 0.0, 1.0, 0.5),
         (48, 70, 40, 0.0, 1.0, 3.0), (40, 60, 36, 62.0, 1.0, 2.0), (33, 45, 36, 60.0, 1.2, 1.2),
         (48, 68, 40, 0.0, 1.3, 1.0), (48, 68, 40, 0.0, 2.5, 1.0), (1, 3, 8, 0.0, 1.0, 1.0), (5, 9, 12, 20.0, 1.0, 1.0)]


def corners(g, c, s, tx, ty):
    """First and last detector position under a tile (tile_corner) and whether it is seen from behind."""
    n, W, P, d, bw, dS = g
    lo, hi, bad = np.full(c.shape, np.inf, F), np.full(c.shape, -np.inf, F), np.zeros(c.shape, bool)
    for ex, ey in ((0, 0), (1, 0), (1, 1), (0, 1)):
        cx, cy = F(1) * (tx * TILE - F(0.5) + F(TILE * ex)), F(1) * (ty * TILE - F(0.5) + F(TILE * ey))
        oc = cx * c + cy * s
        if d > 0:
            qe = cx * s - cy * c + F(d)
            bad |= ~(qe > F(1e-3) * F(d))
            oc = F(d) * oc / qe
        lo, hi = np.minimum(lo, oc), np.maximum(hi, oc)
    return lo, hi, bad


def spans(g, c, s, tx, ty, past):
    n, W, P, d, bw, dS = g
    lo, hi, bad = corners(g, c, s, tx, ty)
    dmax = (W - 1) // 2 + past
    klo = np.maximum(np.floor(np.clip(lo / F(dS), -dmax - 2, dmax + 2)) - 1, -dmax)
    khi = np.minimum(np.ceil(np.clip(hi / F(dS), -dmax - 2, dmax + 2)) + 1, dmax)
    return klo, np.where(bad, 1 << 20, khi - klo + 1)


def square(g, c64, s64, tx, ty, w, seg, klo):
    """square_view: r, E, T, d - v, n, o, whether x's window is the later one."""
    n_, W, P, d, bw, dS = g
    c, s = c64.astype(F), s64.astype(F)
    xw, yw = tx * TILE + (w & 1) * 8 + 3.5, ty * TILE + (w >> 1) * 8 + 3.5
    uc = xw * c64 + yw * s64
    rmax = W // 2 + 128
    if d > 0:
        qd = d - (yw * c64 - xw * s64)
        qec = qd.astype(F)
        cG, invG = F(dS / d), F(d / dS)
        r = np.clip(np.rint(uc.astype(F) * invG / qec), -rmax, rmax)
        T64 = r.astype(np.float64) * dS / d
        T, E = T64.astype(F), (uc - T64 * qd).astype(F)
        qm = np.maximum(qec - F(5), F(1e-3) * F(d))
        G, Gmin = qec * cG, qm * cG
        slack = (F(1.5) * G + F(9) * np.abs(T) + F(9)) / qm
    else:
        r = np.clip(np.rint(uc.astype(F) * F(1 / dS)), -rmax, rmax)
        T, E = np.zeros_like(c), (uc - r.astype(np.float64) * dS).astype(F)
        qec = np.ones_like(c)
        G = Gmin = np.full_like(c, dS)
        slack = np.zeros_like(c)
    kx, ky = c - T * s, s + T * c
    reach = (np.abs(kx) + np.abs(ky) + slack) / Gmin + F(bw) + F(2e-3)
    dlo, dhi = np.abs(kx) / G - slack / Gmin, np.abs(kx) / Gmin + slack / Gmin
    n, o = np.full(c.shape, 1 << 20), np.zeros(c.shape, int)
    for t in range(3):
        need = reach + np.maximum(np.abs(dlo - t), np.abs(dhi - t))
        nt = np.maximum(np.ceil(np.minimum(need, 4096)), 2).astype(int)
        o, n = np.where(nt < n, t, o), np.minimum(n, nt)
    return r, E, T, qec, np.minimum(n, seg - o), o, kx < 0


@pytest.mark.parametrize("g", GEOMS, ids=str)
def test_windows_hold_every_detector(g):
    n, W, P, d, bw, dS = g
    half, dmax, tiles = (n - 1) // 2, (W - 1) // 2, ((n - 1) // 2 + TILE) // TILE
    nv = P if d > 0 else P // 2
    th = ((F(2) * np.arange(nv, dtype=F) * PI_F) / F(P)).astype(np.float64)
    C, S = np.cos(th), np.sin(th)
    widest = 0
    for tx in range(tiles):
        for ty in range(tx + 1):
            widest = max(widest, spans(g, C.astype(F), S.astype(F), F(tx), F(ty), 0)[1].max())
    if widest > 64:
        pytest.skip("the plan takes the unstaged kernel (widest shadow %d)" % widest)
    seg = 32 if widest <= 32 else 64
    rng = np.random.default_rng(n)
    met = 0
    for _ in range(min(40, 4 * tiles * tiles)):
        tx = int(rng.integers(0, tiles))
        ty = int(rng.integers(0, tx + 1))
        i = rng.choice(nv, min(nv, 24), replace=False)
        c, s = C[i], S[i]
        klo, nseg = spans(g, c.astype(F), s.astype(F), F(tx), F(ty), PAST)
        sq = [square(g, c, s, tx, ty, w, seg, klo) for w in range(4)]
        cnt = np.minimum(np.maximum(nseg, np.max([q[4] + q[5] for q in sq], axis=0)), seg + 2 * PAST)
        for w, (r, E, T, qec, nn, o, xlater) in enumerate(sq):
            lo = klo - r
            hi = lo + (cnt - nn - o)
            for pair in range(32):
                dx, dy = F(pair % 4 * 2 - 3), F(pair // 4) - F(3.5)
                du, dv = dx * c.astype(F) + dy * s.astype(F), dy * c.astype(F) - dx * s.astype(F)
                t = E + du
                if d > 0:
                    t = (t + T * dv) * F(d / dS) / (qec - dv)
                else:
                    t = t * F(1 / dS)
                cb = np.rint(np.clip(t - F(0.5) * (nn - 1 + o).astype(F), lo, hi))
                for b in (0, 1):
                    x = tx * TILE + (w & 1) * 8 + int(dx + 3) + b
                    y = ty * TILE + (w >> 1) * 8 + int(dy + 3.5)
                    if x > half or y > x:
                        continue
                    first = r + cb + np.where(xlater == (b == 0), o, 0)
                    u, v = x * c + y * s, y * c - x * s
                    G = dS * (d - v) / d if d > 0 else np.full(c.shape, dS)
                    k = np.rint(u / G)[:, None] + np.arange(-12, 13)[None, :]
                    Tk = k * dS / d if d > 0 else 0.0 * k
                    c_, s_ = c[:, None], s[:, None]
                    meets = np.abs(u[:, None] - k * G[:, None]) < 0.5 * (G[:, None] * bw + np.abs(c_ - Tk * s_) + np.abs(s_ + Tk * c_))
                    meets &= np.abs(k) <= dmax
                    assert not (meets & (np.abs(k) <= dmax))[:, [0, -1]].any() or bw > 1
                    if bw > 1:   # and the detectors of the corner shadow alone
                        if d > 0:
                            ts = np.array([d * ((x + ex) * c + (y + ey) * s) / ((x + ex) * s - (y + ey) * c + d)
                                           for ex, ey in ((-.5, -.5), (.5, -.5), (.5, .5), (-.5, .5))])
                            a, e = ts.min(0) / dS, ts.max(0) / dS
                        else:
                            hw = 0.5 * (np.abs(c) + np.abs(s))
                            a, e = (u - hw) / dS, (u + hw) / dS
                        meets &= (k >= np.round(a)[:, None]) & (k <= np.round(e)[:, None])
                    held = (k >= first[:, None]) & (k < (first + nn)[:, None])
                    staged = (k >= klo[:, None]) & (k < (klo + cnt)[:, None])
                    assert not (meets & ~(held & staged)).any()
                    met += meets.sum()
    assert met > 0
