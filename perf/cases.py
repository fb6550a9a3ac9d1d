"""Performance cases of the engine: the calls a reconstruction program makes, over the sizes it makes
them at.

kinds
  proj    one forward projection and one backprojection (``Projector``), the pair every iterative
          method repeats; fan (d > 0) or parallel beam (d = 0)
  fbp     filtered backprojection of a sinogram (``Projector.fbp``)
  bhc     one density evaluation of the polychromatic model: the likelihood (read by the host, as a
          line search does) and its gradient in the density (``BHCModel``)
  batch   many slices of uneven size, one captured launch per direction (``batch.Batch``)
  tv      the total-variation proximal map (``tv.denoise``)
  admm    the wavelet proximal map (``wavelet.admm``)
  parprj  the double-precision masked parallel operator, both directions (``ctprj_par_*``)
  host    ``setup()`` / ``gpuPrj()`` on ordinary host buffers, as the MEX gateway calls them

``exact`` restates each in double precision with torch alone.
"""
import ctypes
import math

import numpy as np
import torch

import imgrecsrc_b200 as ct
from imgrecsrc_b200 import batch as ctbatch
from imgrecsrc_b200 import bhc as ctbhc
from imgrecsrc_b200 import tv as cttv
from imgrecsrc_b200 import wavelet as ctwvlt

DEV = "cuda"


def _proj(name, n, W, views, full, d, **more):
    return dict(name=name, kind="proj", n=n, W=W, views=views, full=full, d=float(d), **more)


def listed():
    return [
        # the smallest call in use: a 64^2 fan slice (the size of the smoke check), launch-bound
        _proj("fan_64", 64, 90, 48, 48, 200.0),
        # the reference CPU path's parallel-beam workload: 256^2, 180 views over [0, pi)
        _proj("par_256", 256, 363, 180, 360, 0.0),
        # the fan-beam workload of the adjoint and accuracy checks
        _proj("fan_512", 512, 1024, 360, 360, 2048.0),
        # an odd size with an odd detector count, at the view count of a full clinical half turn
        _proj("par_1001", 1001, 1423, 720, 1440, 0.0),
        # the full-size fan workload of the reconstruction loop (the benchmark's step)
        _proj("fan_2048", 2048, 2048, 1440, 1440, 8192.0),
        # direct reconstruction on the polychromatic model's own geometry (source close to the object)
        dict(name="fbp_fan_1024", kind="fbp", n=1024, W=1024, views=720, full=720, d=2048.0),
        # one density evaluation of the polychromatic model at its own configuration, J = 20
        dict(name="bhc_1024", kind="bhc", n=1024, W=1024, views=720, full=720, d=2048.0, J=20),
        # half of the mixed-size batch workload (n of 128 .. 1024, 90 .. 720 views, both beams)
        dict(name="batch_32", kind="batch", count=32, slices_seed=0),
        # the TV map of one regularised density step: 100 inner iterations at 512^2
        dict(name="tv_512", kind="tv", rows=512, cols=512, iters=100, tv="iso"),
        # the default wavelet map (Haar, 6 levels) of one regularised density step at 1024^2
        dict(name="admm_1024", kind="admm", rows=1024, cols=1024, iters=50, daub=2, levels=6),
        # the masked double-precision operator: 512^2 disc, 360 angles over [0, 180)
        dict(name="parprj_512", kind="parprj", n=512, W=727, angles=360),
        # the drop-in entry point on pageable host arrays, forward and back
        dict(name="host_512", kind="host", n=512, W=1024, views=360, full=360, d=2048.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_geometry(rng, lo, hi, fan):
    n = _log_int(rng, lo, hi)
    full = 4 * max(6, int(n * rng.uniform(0.5, 0.7) / 4))
    if fan:
        views = full if rng.random() < 0.7 else int(full * rng.uniform(0.55, 0.95))
        d = float(round(n * rng.choice([2.0, 2.5, 3.0, 4.0])))
    else:
        views, full, d = full, 2 * full, 0.0
    return dict(n=n, W=int(n * rng.uniform(1.0, 1.45)), views=views, full=full, d=d)


def draw(rng):
    kind = rng.choice(["proj", "proj", "proj", "proj", "fbp", "bhc", "batch", "tv", "admm", "parprj", "host"])
    fan = rng.random() < 0.5
    if kind == "proj":
        return dict(kind=kind, **_draw_geometry(rng, 48, 2048, fan))
    if kind == "fbp":
        return dict(kind=kind, **_draw_geometry(rng, 128, 1600, fan))
    if kind == "bhc":
        return dict(kind=kind, J=rng.choice([15, 20, 30]), **_draw_geometry(rng, 128, 1400, fan))
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(4, 28), slices_seed=rng.randint(1, 10000))
    if kind == "tv":
        rows = _log_int(rng, 100, 1500)
        return dict(kind=kind, rows=rows, cols=rows if rng.random() < 0.6 else int(rows * rng.uniform(0.7, 1.3)),
                    iters=rng.choice([20, 50, 100]), tv=rng.choice(["iso", "iso", "l1"]))
    if kind == "admm":
        return dict(kind=kind, rows=64 * rng.randint(2, 24), cols=64 * rng.randint(2, 24),
                    iters=rng.choice([20, 50]), daub=rng.choice([2, 2, 2, 6]), levels=rng.randint(4, 6))
    if kind == "parprj":
        n = _log_int(rng, 64, 600)
        return dict(kind=kind, n=n, W=int(1.42 * n), angles=rng.randint(max(30, n // 2), n))
    return dict(kind="host", **_draw_geometry(rng, 64, 1024, fan))


# ------------------------------------------------------------------- inputs

def _geometry(c):
    return ct.Geometry(c["n"], c["W"], c["views"], c["full"], 1.0, 1.0, c["d"])


def _ellipses(rng, count, lo, hi):
    r, t = np.sqrt(rng.uniform(0, 1, count)), rng.uniform(0, 2 * np.pi, count)
    return [dict(cx=r[i] * np.cos(t[i]) * 0.6, cy=r[i] * np.sin(t[i]) * 0.6, a=rng.uniform(0.05, 0.3),
                 b=rng.uniform(0.05, 0.3), phi=rng.uniform(0, np.pi), v=rng.uniform(lo, hi)) for i in range(count)]


def _image(n, ells):
    """Sum of ellipses on the n x n grid (unit square [-1, 1]^2), on the GPU, float64."""
    c = (torch.arange(n, device=DEV, dtype=torch.float64) - n // 2) / (n / 2.0)
    X, Y = c[None, :], c[:, None]
    img = torch.zeros(n, n, device=DEV, dtype=torch.float64)
    for e in ells:
        cp, sp = math.cos(e["phi"]), math.sin(e["phi"])
        u = (X - e["cx"]) * cp + (Y - e["cy"]) * sp
        v = -(X - e["cx"]) * sp + (Y - e["cy"]) * cp
        img += e["v"] * ((u / e["a"]) ** 2 + (v / e["b"]) ** 2 <= 1.0)
    return img


def _phantom(n, seed):
    rng = np.random.default_rng(seed)
    return _image(n, _ellipses(rng, 10, -0.5, 1.0)).clamp_(min=0.0).float()


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _noise(shape, seed, scale=1.0):
    return torch.randn(shape, device=DEV, generator=_gen(seed)) * scale


def _line_integrals(c, ells):
    """Closed-form line integrals of the ellipses along every ray (pixel units)."""
    n, W, npv, P, d = c["n"], c["W"], c["views"], c["full"], c["d"]
    t = torch.arange(W, device=DEV, dtype=torch.float64) - W // 2
    B = torch.atan(t / d) if d > 0 else torch.zeros_like(t)
    off = (t * torch.cos(B))[None, :]
    R = (2 * math.pi / P) * torch.arange(npv, device=DEV, dtype=torch.float64)[:, None] + B[None, :]
    s, h = torch.zeros(npv, W, device=DEV, dtype=torch.float64), n / 2.0
    for e in ells:
        al = R - e["phi"]
        a, b = e["a"] * h, e["b"] * h
        r2 = (a * torch.cos(al)) ** 2 + (b * torch.sin(al)) ** 2
        q = off - h * (e["cx"] * torch.cos(R) + e["cy"] * torch.sin(R))
        s += e["v"] * 2 * a * b * torch.sqrt((r2 - q * q).clamp(min=0.0)) / r2
    return s


FOV_CM, I0 = 2.0, 1e5    # field of view and photons per ray of the polychromatic workload


def _bhc_inputs(c, seed):
    rng = np.random.default_rng(seed)
    J = c["J"]
    ells = [dict(cx=0.0, cy=0.0, a=rng.uniform(0.6, 0.8), b=rng.uniform(0.5, 0.7), phi=rng.uniform(0, np.pi), v=2.7)]
    ells += _ellipses(rng, 8, 0.5, 5.1)
    x = _image(c["n"], ells)
    mu, sig = rng.uniform(0.35, 0.65) * (J - 1), rng.uniform(0.08, 0.15) * J
    Ie = np.exp(-0.5 * ((np.arange(J) - mu) / sig) ** 2) + 1e-3
    Ie = torch.from_numpy(Ie / Ie.sum()).to(DEV)
    BL, _ = _b1_out(FOV_CM / c["n"] * _line_integrals(c, ells), _nodes(J), Ie)
    m = (torch.poisson(I0 * BL, generator=_gen(seed)) / I0).float()
    # the current iterate: the object with 5 % of local error
    x = (x * (1.0 + 0.05 * _noise(x.shape, seed + 1).double())).float()
    return x, Ie, m


def prepare(c, seed):
    kind, seed = c["kind"], int(seed)
    if kind in ("proj", "fbp"):
        pr = ct.Projector(_geometry(c))
        st = dict(kind=kind, pr=pr, y=_noise(pr.sino_shape, seed), b=torch.empty(pr.img_shape, device=DEV))
        if kind == "proj":
            st.update(x=_phantom(c["n"], seed), s=torch.empty(pr.sino_shape, device=DEV))
        return st
    if kind == "bhc":
        x, Ie, m = _bhc_inputs(c, seed)
        pr = ct.Projector(_geometry(c))
        model = ctbhc.BHCModel(pr, ctbhc.kappa_nodes(c["J"]), FOV_CM / c["n"])
        return dict(kind=kind, pr=pr, model=model, x=x, Ie=Ie, m=m)
    if kind == "batch":
        geoms = ctbatch.cfg4_geometries(c["count"], c["slices_seed"])
        imgs = [_phantom(g.n, seed + i) for i, g in enumerate(geoms)]
        ys = [_noise((g.np, g.prjWidth), seed + 1000 + i) for i, g in enumerate(geoms)]
        sinos = [torch.empty(g.np, g.prjWidth, device=DEV) for g in geoms]
        backs = [torch.empty(g.n, g.n, device=DEV) for g in geoms]
        b = ctbatch.Batch(geoms)
        b.bind(imgs, sinos, ys, backs)
        b.capture()
        return dict(kind=kind, b=b, out=dict(sinos=sinos, backs=backs), keep=(imgs, ys))
    if kind in ("tv", "admm"):
        n = max(c["rows"], c["cols"])
        x = _phantom(n, seed)[: c["rows"], : c["cols"]].contiguous()
        x += _noise(x.shape, seed + 1, 0.1)
        st = dict(kind=kind, x=x, c=dict(c))
        if kind == "admm":
            st["h"] = ctwvlt.daubcqf(c["daub"])
        return st
    if kind == "parprj":
        mask, theta = _par_mask(c["n"]), _par_theta(c)
        conf = ct._lib.ParDevConf(1.0, c["n"], c["n"], c["angles"], c["W"])
        x = torch.rand(mask.numel(), dtype=torch.float64, device=DEV, generator=_gen(seed))
        y = torch.randn(c["angles"] * c["W"], dtype=torch.float64, device=DEV, generator=_gen(seed + 1))
        return dict(kind=kind, conf=conf, theta=theta, mask=mask.double(), x=x, y=y)
    g = _geometry(c)
    ct.lib().setup(g.n, g.prjWidth, g.np, g.prjFull, g.dSize, g.effectiveRate, g.d)
    return dict(kind=kind, x=_phantom(g.n, seed).cpu().numpy(), y=_noise((g.np, g.prjWidth), seed).cpu().numpy(),
                s=np.zeros((g.np, g.prjWidth), np.float32), b=np.zeros((g.n, g.n), np.float32))


def run(st):
    kind = st["kind"]
    if kind == "proj":
        return dict(s=st["pr"].forward(st["x"], out=st["s"]), b=st["pr"].backward(st["y"], out=st["b"]))
    if kind == "fbp":
        return st["pr"].fbp(st["y"], out=st["b"])
    if kind == "bhc":
        f = st["model"].forward(st["x"], st["Ie"], st["m"])
        gx, _ = st["model"].backward(grad_Ie=False)
        return dict(f=f.item(), gx=gx)
    if kind == "batch":
        st["b"].forward()
        st["b"].backward()
        return st["out"]
    if kind == "tv":
        c = st["c"]
        X, it = cttv.denoise(st["x"], 0.05, 0.0, c["iters"], tv_type=c["tv"], n_row=c["cols"], n_col=c["rows"])
        return dict(x=X, iterations=it)
    if kind == "admm":
        c = st["c"]
        a, it = ctwvlt.admm(st["x"], 0.05, st["h"], c["levels"], 0.0, c["iters"])
        return dict(a=a, iterations=it)
    L, vp = ct.lib(), lambda t: ctypes.c_void_p(t.data_ptr())
    if kind == "parprj":
        conf, hs = ctypes.byref(st["conf"]), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        npix = st["mask"].numel()
        s, b = torch.zeros_like(st["y"]), torch.zeros_like(st["x"])
        ct.check(L.ctprj_par_forward(conf, st["theta"].ctypes.data, vp(st["mask"]), npix, vp(st["x"]), vp(s), hs))
        ct.check(L.ctprj_par_backward(conf, st["theta"].ctypes.data, vp(st["mask"]), npix, vp(st["y"]), vp(b), hs))
        return dict(s=s, b=b)
    ct.check(L.gpuPrj(st["x"].ctypes.data, st["s"].ctypes.data, bytes([ct.FWD_BIT])))
    ct.check(L.gpuPrj(st["b"].ctypes.data, st["y"].ctypes.data, bytes([ct.BWD_BIT])))
    return dict(s=st["s"], b=st["b"])


def work(c):
    kind = c["kind"]
    if kind in ("tv", "admm"):
        px = c["rows"] * c["cols"]
        return dict(bytes=8.0 * px, flops=(30.0 if kind == "tv" else 20.0) * px * c["iters"])
    if kind == "batch":
        gs = ctbatch.cfg4_geometries(c["count"], c["slices_seed"])
        return dict(bytes=sum(8.0 * (g.n * g.n + g.np * g.prjWidth) for g in gs),
                    flops=sum(2 * 4.4 * g.n * g.n * g.np for g in gs))
    if kind == "parprj":
        px = 0.73 * c["n"] ** 2
        return dict(bytes=16.0 * (px + c["angles"] * c["W"]), flops=2 * 4.4 * px * c["angles"])
    # a pixel meets about 2.2 detectors per view, one multiply-add each
    px, rays = c["n"] ** 2, c["views"] * c["W"]
    passes = 1 if kind == "fbp" else 2
    flops = passes * 4.4 * px * c["views"] + (30.0 * c["J"] * rays if kind == "bhc" else 0.0)
    return dict(bytes=passes * 4.0 * (px + rays), flops=flops)


# ------------------------------------------------- double-precision restatement

F64 = torch.float64
PI_F = np.float32(3.14159265359)


def _base_angle(i, P):
    """Angle of base view i: formed in single precision, as the interface defines it."""
    return float(np.float32(np.float32(2 * i) * PI_F) / np.float32(P))


def _view_of(j, b, P):
    """Sinogram row of symmetric image j of base view b."""
    return ((0, 1, 2, 3, 2, 3, 4, 1)[j] * (P // 4) + (1 if j < 4 else -1) * b) % P


# the eight images (gx, gy) of pixel (x, y)
_IMAGES = [lambda x, y: (x, y), lambda x, y: (-y, x), lambda x, y: (-x, -y), lambda x, y: (y, -x),
           lambda x, y: (x, -y), lambda x, y: (y, x), lambda x, y: (-x, y), lambda x, y: (-y, -x)]


def _overlap(dist, hb, cR, sR):
    """Overlap of a beam of half width hb at signed distance dist with a unit pixel seen along (cR, sR)."""
    hi, lo = torch.maximum(cR.abs(), sR.abs()), torch.minimum(cR.abs(), sR.abs())
    b2, b1 = 0.5 * (hi + lo), 0.5 * (hi - lo)
    iw = torch.where(lo > 1e-14, 0.5 / lo.clamp(min=1e-14), torch.zeros_like(lo))

    def area(u):
        p = (u + b2).clamp(min=0.0).minimum(lo)
        r = (u - b1).clamp(min=0.0).minimum(lo)
        return (p * p - r * r) * iw + (u + b1).clamp(min=0.0).minimum(2 * b1) + r
    return (area(hb - dist) - area(-hb - dist)) / hi


def _chunks(count, elems):
    step = max(1, min(count, int((1 << 22) // max(1, elems))))
    return [range(i, min(count, i + step)) for i in range(0, count, step)]


def _col(v):
    return torch.tensor(v, device=DEV, dtype=F64)


def _forward64(c, img):
    n, W, npv, P, d = c["n"], c["W"], c["views"], c["full"], c["d"]
    half, h2, pC = (n - 1) // 2, n // 2, W // 2
    k0 = 1 - W % 2
    k = torch.arange(k0, W, device=DEV)
    t = (k - pC).to(F64)
    bq = torch.sqrt(t * t + d * d) if d > 0 else torch.ones_like(t)
    cB, sB = (d / bq, t / bq) if d > 0 else (torch.ones_like(t), torch.zeros_like(t))
    off = (t * cB)[None, :, None]
    y = torch.arange(-half, half + 1, device=DEV)
    yd = y.to(F64)[None, None, :]
    src = img.to(F64).reshape(-1)
    out = torch.zeros(npv, W, device=DEV, dtype=F64)
    for bs in _chunks(min(npv, P // 8 + 1), k.numel() * y.numel()):
        th = [_base_angle(b, P) for b in bs]
        cT, sT = _col([math.cos(a) for a in th])[:, None, None], _col([math.sin(a) for a in th])[:, None, None]
        cR, sR = cB[None, :, None] * cT - sB[None, :, None] * sT, sB[None, :, None] * cT + cB[None, :, None] * sT
        x0 = torch.round((off - yd * sR) / cR).long()
        S = [torch.zeros(len(bs), k.numel(), device=DEV, dtype=F64) for _ in range(8)]
        for q in range(-3, 4):
            x = x0 + q
            dist = x * cR + yd * sR - off
            hb = 0.5 * (1.0 + (x * sT - yd * cT) / d) * cB[None, :, None] if d > 0 else torch.full_like(dist, 0.5)
            w = _overlap(dist, hb, cR, sR) * (x.abs() <= half)
            x = x.clamp(-half, half)
            yb = y[None, None, :].expand_as(x)
            for j in range(8):
                gx, gy = _IMAGES[j](x, yb)
                S[j] += (w * src[(gy + h2) * n + gx + h2]).sum(dim=2)
        for i, b in enumerate(bs):
            for j in range(8):
                v = _view_of(j, b, P)
                if v < npv and (j < 4 or 0 < b < P / 8):
                    out[v, k if j < 4 else 2 * pC - k] = S[j][i]
    return out


def _backward64(c, sino, fbp=False):
    n, W, npv, P, d = c["n"], c["W"], c["views"], c["full"], c["d"]
    half, h2, pC, dmax = (n - 1) // 2, n // 2, W // 2, (W - 1) // 2
    xs, ys = torch.meshgrid(torch.arange(half + 1, device=DEV), torch.arange(half + 1, device=DEV), indexing="ij")
    keep = ys <= xs
    xs, ys = xs[keep], ys[keep]
    xd, yd = xs.to(F64)[None, :], ys.to(F64)[None, :]
    src = torch.cat([sino.to(F64).reshape(-1), torch.zeros(W, device=DEV, dtype=F64)])   # row npv: absent views
    S = [torch.zeros(xs.numel(), device=DEV, dtype=F64) for _ in range(8)]
    for vs in _chunks(P if d > 0 else P // 2, xs.numel()):
        th = [_base_angle(i, P) for i in vs]
        cT, sT = _col([math.cos(a) for a in th])[:, None], _col([math.sin(a) for a in th])[:, None]
        u, v = xd * cT + yd * sT, yd * cT - xd * sT
        qe = d - v
        k0 = torch.round(d * u / qe if d > 0 else u).long()
        rows = [[min(npv, _view_of(j, i, P)) for i in vs] for j in range(8)]
        rows2 = [[min(npv, (_view_of(j, i, P) + P // 2) % P) for i in vs] for j in range(8)]
        rows, rows2 = [[torch.tensor(r, device=DEV)[:, None] * W for r in q] for q in (rows, rows2)]
        for q in range(-3, 4):
            k = k0 + q
            t = k.to(F64)
            if d > 0:
                bq = torch.sqrt(t * t + d * d)
                cB, sB = d / bq, t / bq
                w = _overlap(cB * (u - t) + sB * v, 0.5 * qe * cB / d, cB * cT - sB * sT, sB * cT + cB * sT)
                if fbp:
                    w = w * (d / qe) ** 2
            else:
                w = _overlap(u - t, torch.full_like(u, 0.5), cT, sT)
            w = w * (k.abs() <= dmax)
            k = k.clamp(-dmax, dmax)
            for j in range(8):
                kj = k if j < 4 else -k
                S[j] += (w * src[rows[j] + pC + kj]).sum(dim=0)
                if d <= 0:
                    S[j] += (w * src[rows2[j] + pC - kj]).sum(dim=0)
    img = torch.zeros(n, n, device=DEV, dtype=F64)
    for j in range(7, -1, -1):    # pixels on an axis or a diagonal have four distinct images: 0..3
        gx, gy = _IMAGES[j](xs, ys)
        use = slice(None) if j < 4 else (ys > 0) & (ys < xs)
        img[(gy + h2)[use], (gx + h2)[use]] = S[j][use]
    return img


def _fbp64(c, sino):
    W, d, N = c["W"], c["d"], 2 * c["W"]
    x = sino.to(F64)
    if d > 0:
        t = torch.arange(W, device=DEV, dtype=F64) - W // 2
        x = x * (d / torch.sqrt(d * d + t * t))
    i = np.arange(1, N, 2)
    m = np.where(i < N / 2, i, N - i).astype(np.float32)
    ramp = np.zeros(N)
    ramp[0] = 0.25
    ramp[i] = np.float32(np.float32(np.float32(-1.0) / PI_F) / PI_F) / m / m
    arg = (np.float32(2.0) * PI_F * np.arange(N).astype(np.float32)) / np.float32(N)
    H = np.fft.fft(ramp).real * (0.5 + 0.5 * np.cos(arg.astype(np.float64)))
    H = torch.from_numpy(H).to(DEV)
    y = torch.fft.ifft(torch.fft.fft(x, n=N, dim=1) * H, dim=1).real[:, :W]
    return _backward64(c, y, fbp=True) * float(PI_F / np.float32(c["views"]))


def _nodes(J, kmin=1e-2, kmax=1e2):
    k = np.logspace(math.log10(kmin), math.log10(kmax), J)
    q = k[1] / k[0]
    return np.concatenate([[k[0] / q], k, [k[-1] * q]])


def _b1_out(s, k, Ie):
    """(BL, dBL/ds) of the degree-1 spline spectrum model: exact transforms of the hat functions, and
    near s = 0 the cubic expansions that define the model there."""
    BL, sBL = torch.zeros_like(s), torch.zeros_like(s)
    for j in range(len(k) - 2):
        a, b, c = (float(v) for v in k[j:j + 3])
        eL, eC, eR = torch.exp(-a * s), torch.exp(-b * s), torch.exp(-c * s)
        # divided differences of powers: (a^m - b^m) / (a - b) - (b^m - c^m) / (b - c)
        D = [(a ** m - b ** m) / (a - b) - (b ** m - c ** m) / (b - c) for m in range(7)]
        co = [-D[2] / 2, D[3] / 6, -D[4] / 24, D[5] / 120]
        dc = [D[3] / 6, -D[4] / 12, D[5] / 40, -D[6] / 180]
        v = -(eL - eC) / (s * s * (a - b)) + (eC - eR) / (s * s * (b - c))
        near = s.abs() < abs(1e-6 * co[0] / co[3]) ** (1 / 3)
        v = torch.where(near, co[0] + s * (co[1] + s * (co[2] + s * co[3])), v)
        w = (2 * (eL - eC) / (s ** 3 * (a - b)) + (a * eL - b * eC) / (s * s * (a - b))
             - 2 * (eC - eR) / (s ** 3 * (b - c)) - (b * eC - c * eR) / (s * s * (b - c)))
        near = s.abs() < abs(1e-6 * dc[0] / dc[3]) ** (1 / 3)
        w = torch.where(near, dc[0] + s * (dc[1] + s * (dc[2] + s * dc[3])), w)
        BL += Ie[j] * v
        sBL += Ie[j] * w
    return BL, sBL


def _bhc64(c, seed):
    x, Ie, m = _bhc_inputs(c, seed)
    Ts, m = FOV_CM / c["n"], m.double()
    BL, sBL = _b1_out(Ts * _forward64(c, x), _nodes(c["J"]), Ie)
    f = (BL - m - torch.where(m > 0, m * torch.log(BL / m.clamp(min=1e-30)), torch.zeros_like(m))).sum()
    return dict(f=f.item(), gx=Ts * _backward64(c, (1 - m / BL) * sBL))


def _tv64(X, lam, iters, kind):
    D, t = torch.zeros_like(X), 1.0
    P = [torch.zeros_like(X), torch.zeros_like(X)]   # vertical, horizontal; last row / column zero
    R, f = [p.clone() for p in P], math.inf
    for _ in range(iters):
        L = R[0] + R[1]
        L[1:] -= R[0][:-1]
        L[:, 1:] -= R[1][:, :-1]
        C = X - lam * L
        D = C.clamp(min=0.0)
        Q = [torch.zeros_like(X), torch.zeros_like(X)]
        Q[0][:-1] = D[:-1] - D[1:]
        Q[1][:, :-1] = D[:, :-1] - D[:, 1:]
        N = [r + q / (8 * lam) for r, q in zip(R, Q)]
        if kind == "iso":
            s = torch.sqrt((N[0] ** 2 + N[1] ** 2).clamp(min=1.0))
            N = [v / s for v in N]
        else:
            N = [v.clamp(-1.0, 1.0) for v in N]
        t1 = 0.5 * (1 + math.sqrt(1 + 4 * t * t))
        R = [v + (t - 1) / t1 * (v - p) for v, p in zip(N, P)]
        P, fold = N, f
        f = float((C ** 2).sum() - ((C - D) ** 2).sum())
        t = 1.0 if f > fold else t1
    return D


def _split(x, h, g, dim):
    idx = 2 * torch.arange(x.shape[dim] // 2, device=x.device)
    take = [x.index_select(dim, (idx + j) % x.shape[dim]) for j in range(len(h))]
    return torch.cat([sum(f[j] * take[j] for j in range(len(h))) for f in (h, g)], dim)


def _join(x, h, g, dim):
    m = x.shape[dim] // 2
    lo, hi = x.narrow(dim, 0, m), x.narrow(dim, m, m)
    out, idx = torch.zeros_like(x), 2 * torch.arange(m, device=x.device)
    for j in range(len(h)):
        out.index_add_(dim, (idx + j) % (2 * m), h[j] * lo + g[j] * hi)
    return out


def _dwt64(x, h, levels, inverse=False):
    g = [(-1) ** j * h[len(h) - 1 - j] for j in range(len(h))]
    y = x.clone()
    for lev in (range(levels - 1, -1, -1) if inverse else range(levels)):
        r, c = x.shape[0] >> lev, x.shape[1] >> lev
        blk = y[:r, :c].clone()
        y[:r, :c] = _join(_join(blk, h, g, 0), h, g, 1) if inverse else _split(_split(blk, h, g, 1), h, g, 0)
    return y


def _admm64(a, u, h, levels, iters):
    nu, rho, cnt = torch.zeros_like(a), 1.0, 0
    s = _dwt64(a, h, levels)
    for _ in range(iters + 1):
        cnt += 1
        al = ((a + rho * _dwt64(s + nu, h, levels, True)) / (1 + rho)).clamp(min=0.0)
        v, old = _dwt64(al, h, levels), s
        w = v - nu
        s = torch.sign(w) * (w.abs() - u / rho).clamp(min=0.0)
        nu = nu + s - v
        dif, res = float((s - old).norm()), float((s - v).norm())
        if cnt > 20 and _ < iters:
            if dif > 10 * res:
                rho, nu, cnt = rho / 2, nu * 2, 0
            elif dif < res / 10:
                rho, nu, cnt = rho * 2, nu / 2, 0
    return ((a + rho * _dwt64(s + nu, h, levels, True)) / (1 + rho)).clamp(min=0.0)


def _daub64(taps):
    """Minimum-phase Daubechies scaling filters of 2 and 6 taps, in closed form."""
    if taps == 2:
        return [math.sqrt(0.5)] * 2
    p, q = math.sqrt(10.0), math.sqrt(5 + 2 * math.sqrt(10.0))
    v = [1 + p + q, 5 + p + 3 * q, 10 - 2 * p + 2 * q, 10 - 2 * p - 2 * q, 5 + p - 3 * q, 1 + p - q]
    return [x * math.sqrt(2.0) / 32 for x in v]


def _par_mask(n):
    """0-based column-major indices of a disc of radius 0.48 n."""
    r = torch.arange(n, device=DEV, dtype=F64) - (n - 1) / 2
    return torch.nonzero(((r[:, None] ** 2 + r[None, :] ** 2) <= (0.48 * n) ** 2).t().reshape(-1)).squeeze(1)


def _par_theta(c):
    return np.ascontiguousarray(np.arange(c["angles"]) * 180.0 / c["angles"])


def _parprj64(c, x, y):
    n, W, pC, pi = c["n"], c["W"], c["n"] // 2, 3.14159265
    m = _par_mask(n)
    px, py = (m // n - pC).to(F64), (m % n - pC).to(F64)
    s, b, yr = torch.zeros(c["angles"], W, device=DEV, dtype=F64), torch.zeros_like(x), y.reshape(-1, W)
    for it, th in enumerate(_par_theta(c)):
        tmp = abs(int(math.fmod(th, 90) - 45)) * pi / 180     # the footprint's angle is in whole degrees
        H, b1, b2 = 1 / math.sin(tmp + pi / 4), math.sqrt(0.5) * math.sin(tmp), math.sqrt(0.5) * math.cos(tmp)
        w, dist = b2 - b1, px * math.cos(th * pi / 180) + py * math.sin(th * pi / 180)
        lb, ub = torch.ceil(dist - b2 - 0.5 + 1e-8), torch.floor(dist + b2 + 0.5 - 1e-8)

        def area(u):   # of the trapezoid up to u
            p, r = (u + b2).clamp(0.0, w), (u - b1).clamp(0.0, w)
            return H * ((p * p - r * r) * 0.5 / w + (u + b1).clamp(0.0, 2 * b1) + r)
        for q in range(4):
            k = lb + q
            ul, ur = k - 0.5 - dist, k + 0.5 - dist
            v = area(ur) - area(ul)
            # both edges on one ramp: the midpoint height; left edge on the falling ramp likewise
            v = torch.where((ul > -b2) & (ur <= -b1), H / w * (k - dist + b2), v)
            v = torch.where((ul > b1) & (ur <= b2), H / w * (dist + b2 - k), v)
            ok = (k <= ub) & (k >= -pC) & (k + pC < min(n, W))
            kk = (k + pC).clamp(0, W - 1).long()
            v = torch.where(ok, v, torch.zeros_like(v))
            s[it].index_add_(0, kk, v * x)
            b += v * yr[it][kk]
    return dict(s=s.reshape(-1), b=b)


def exact(c, seed):
    kind, seed = c["kind"], int(seed)
    if kind in ("proj", "host"):
        shape = (c["views"], c["W"])
        return dict(s=_forward64(c, _phantom(c["n"], seed)), b=_backward64(c, _noise(shape, seed)))
    if kind == "fbp":
        return _fbp64(c, _noise((c["views"], c["W"]), seed))
    if kind == "bhc":
        return _bhc64(c, seed)
    if kind == "batch":
        out = dict(sinos=[], backs=[])
        for i, g in enumerate(ctbatch.cfg4_geometries(c["count"], c["slices_seed"])):
            gc = dict(n=g.n, W=g.prjWidth, views=g.np, full=g.prjFull, d=g.d)
            out["sinos"].append(_forward64(gc, _phantom(g.n, seed + i)))
            out["backs"].append(_backward64(gc, _noise((g.np, g.prjWidth), seed + 1000 + i)))
        return out
    if kind in ("tv", "admm"):
        x = _phantom(max(c["rows"], c["cols"]), seed)[: c["rows"], : c["cols"]].contiguous()
        x = (x + _noise(x.shape, seed + 1, 0.1)).double()
        if kind == "tv":
            return dict(x=_tv64(x, 0.05, c["iters"], c["tv"]), iterations=None)
        return dict(a=_admm64(x, 0.05, _daub64(c["daub"]), c["levels"], c["iters"]), iterations=None)
    npix = _par_mask(c["n"]).numel()
    x = torch.rand(npix, dtype=F64, device=DEV, generator=_gen(seed))
    y = torch.randn(c["angles"] * c["W"], dtype=F64, device=DEV, generator=_gen(seed + 1))
    return _parprj64(c, x, y)
