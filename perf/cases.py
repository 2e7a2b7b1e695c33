"""The work a simulation has this package do, as timed cases.

Each case is one call (or one step's calls) through the public entry points:
the wavefront-sensor frame of maos_b200.shwfs.Context with its gradients read
to the host, the stage calls on device buffers, and the science evaluation.
Sizes are those of maos_b200.configs, the tests and the serving simulations,
or lie between them.

Frames run without detector noise, because a photon count is a step function
of its mean; the noise is a case of its own on fixed intensities.
"""
from __future__ import annotations

import functools
import json
import math

import numpy as np
import torch

from maos_b200 import configs, shwfs
from maos_b200.setup import Setup, aperture

AS2RAD = configs.AS2RAD
R0, L0 = 0.186, 30.0
HT = [0.0, 500.0, 1e3, 2e3, 4e3, 8e3, 16e3]
WT = [0.596, 0.0386, 0.0386, 0.0386, 0.1436, 0.0386, 0.1024]
DT = 1.0 / 800
DEV = "cuda"


def listed():
    lgs30 = dict(star="lgs", D=30.0, order=60, nwfs=6, nopd=16, notf=32, pix=6, pixas=1.0, grad="mf", form="fft",
                 layers=7, nx=2048, sdx=1 / 32)
    return [
        # the smallest frame in use: one natural star on an 8 m telescope, where launches and the wait dominate
        dict(name="ngs8_frame", kind="frame", star="ngs", D=8.0, order=16, nwfs=1, nopd=16, notf=32, pix=8, pixas=0.5,
             grad="cog", form="fft", layers=2, nx=1024, sdx=1 / 32),
        # one of the simulations a server runs: 10 m, 64-point transforms, a sampling unrelated to the screens'
        dict(name="ngs10_f64_frame", kind="frame", star="ngs", D=10.0, order=32, nwfs=3, nopd=32, notf=64, pix=8,
             pixas=0.23, grad="cog", form="fft", layers=5, nx=1024, sdx=1 / 32),
        # the frame of a 30 m laser tomography system, in both imaging forms
        dict(lgs30, name="lgs30_frame", kind="frame"),
        dict(lgs30, name="lgs30_frame_tc", kind="frame", form="tc"),
        # its step in closed loop: new mirror surfaces, tip/tilt and focus for every frame
        dict(lgs30, name="lgs30_loop", kind="loop"),
        # the same sensors at twice the sampling: 64-point transforms, long spots, screens larger than the cache
        dict(lgs30, name="lgs30_f64_frame", kind="frame", nopd=32, notf=64, pix=12, pixas=0.8, grad="cog", nx=4096,
             sdx=1 / 64),
        # sensors of three sizes in one frame, launched as a graph
        dict(lgs30, name="uneven_batch", kind="batch"),
        # few, finely sampled subapertures of a truth sensor, from phase that the caller has on the device
        dict(name="ngs30_f128_images", kind="images", star="ngs", D=30.0, order=8, nwfs=1, nopd=64, notf=128, pix=16,
             pixas=0.02, grad="cog", form="fft", layers=3, nx=1024, sdx=1 / 16),
        # one laser sensor's images and gradients from phase that the caller has on the device
        dict(lgs30, name="lgs30_images", kind="images", nwfs=1, layers=3, nx=1024, sdx=1 / 16),
        # geometric sensing, as in the frames of a run before physical optics begin
        dict(lgs30, name="lgs30_ztilt", kind="geom"),
        # a short science exposure: wavefront error of every frame, the point-spread functions at its end
        dict(name="science30", kind="science", D=30.0, sdx=1 / 64, nx=4096, layers=7, dirs=3, wvls=3, nembed=4096,
             psfsize=256, frames=4, pttr=0),
        # photon and read noise on the intensities of the 30 m system's sensors
        dict(name="noise", kind="noise", n=6 * 2820 * 36, mean=14.0, bkgrnd=0.5, rne=3.0),
    ]


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "frame", "loop", "images", "images", "geom", "science", "noise"])
    if kind == "noise":
        return dict(kind=kind, n=int(math.exp(rng.uniform(math.log(1e3), math.log(2e6)))),
                    mean=round(math.exp(rng.uniform(math.log(0.5), math.log(400.0))), 2),
                    bkgrnd=round(rng.uniform(0.0, 5.0), 2), rne=round(rng.uniform(0.0, 6.0), 2))
    if kind == "science":
        ng = rng.choice([512, 1024, 2048, 4096])
        sdx = rng.choice([1 / 32, 1 / 64])
        # at least 4 m, and at most half of the transform
        D = min(30.0, round(rng.uniform(0.3, 0.5) * ng * sdx, 2))
        return dict(kind=kind, D=D, sdx=sdx, nx=1024, layers=rng.randint(1, 7), dirs=rng.randint(1, 5),
                    wvls=rng.randint(1, 3), nembed=ng, psfsize=2 * rng.randint(24, 160), frames=rng.randint(1, 4),
                    pttr=rng.randint(0, 1))
    c = dict(kind=kind, star=rng.choice(["ngs", "lgs"]), nwfs=rng.randint(1, 6), layers=rng.randint(1, 7),
             nx=rng.choice([512, 1024, 2048]), sdx=rng.choice([1 / 16, 1 / 32]), form="fft", grad="cog")
    notf = rng.choice([32, 32, 64])
    if kind == "images":
        c["nwfs"] = 1
        notf = rng.choice([32, 64, 128, 256])
        c["sdx"], c["nx"] = 1 / 16, 1024
    order = int(round(math.exp(rng.uniform(math.log(5.0), math.log(60.0)))))
    if notf >= 128:
        c["star"] = "ngs"
        order = rng.randint(1, 10) if notf == 128 else rng.randint(1, 3)
    dsa = 0.5 if c["star"] == "lgs" else rng.uniform(0.25, 0.8)
    c.update(order=order, D=round(order * dsa, 3), nopd=notf // 2, notf=notf,
             pix=rng.randint(4, 11) if notf == 32 else rng.randint(6, 16),
             pixas=round(rng.uniform(0.6, 1.1) if c["star"] == "lgs" else rng.uniform(0.1, 0.6), 3))
    if notf == 32:
        c["grad"] = rng.choice(["cog", "mf"])
        if c["pix"] <= 8:
            c["form"] = rng.choice(["fft", "fft", "tc"])
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _config(c):
    """The powfs configuration of a case, in the vocabulary of maos_b200.configs."""
    lgs = c["star"] == "lgs"
    dsa = c["D"] / c["order"]
    n = c["nwfs"]
    rad = 35.0 if lgs else 20.0
    ang = [2 * math.pi * k / n for k in range(n)]
    one = n == 1 and not lgs
    cfg = dict(name=c["kind"], D=c["D"], Din=0.12 * c["D"], amp_binary=0, order=c["order"], dsa=dsa, dx=dsa / c["nopd"],
               saat=0.3, embfac=c["notf"] // c["nopd"], notf=c["notf"], pixpsa=c["pix"], pixtheta=c["pixas"] * AS2RAD,
               pixblur=0.3, wvl=0.589e-6 if lgs else 0.7e-6, hs=90e3 if lgs else math.inf,
               siglev=500.0 if lgs else 1000.0, rne=3.0, bkgrnd=0.0, bkgrndc=0.0,
               phytype=1 if c["grad"] == "mf" else 2, sigmatch=1, mtchcr=1 if c["grad"] == "mf" and lgs else 0,
               cogthres=0.0, cogoff=0.0, r0=R0, L0=L0, has_llt=0, nwfs=n,
               thetax=[0.0 if one else rad * AS2RAD * math.cos(a) for a in ang],
               thetay=[0.0 if one else rad * AS2RAD * math.sin(a) for a in ang])
    if lgs:
        cfg.update(has_llt=1, llt_d=0.4, llt_widthp=0.6, llt_ox=c["D"] * 4 / 15, llt_oy=0.0,
                   sodium=dict(centers=[90e3], fwhms=[10e3], weights=[1.0]))
    return cfg


def _members(c):
    """The powfs of a case: itself, or with the small sensors of the uneven batch beside it."""
    return [_config(c)] + ([configs.NGS30_2X2, configs.TT30] if c["kind"] == "batch" else [])


@functools.lru_cache(maxsize=None)
def _setup_of(text):
    return Setup({k: math.inf if v == "inf" else v for k, v in json.loads(text).items()})


def _setup(cfg):
    """The host setup of a configuration, made once per process as a program does."""
    return _setup_of(json.dumps({k: "inf" if v == math.inf else v for k, v in cfg.items() if k != "name"}, sort_keys=True))


def _layers(c, seed):
    """Layer descriptors with seeded winds, and the frame index."""
    rng = np.random.default_rng(seed)
    n, dx, nl = c["nx"], c["sdx"], c["layers"]
    wt = np.asarray(WT[:nl]) / sum(WT[:nl])
    v, a = rng.uniform(5.0, 15.0, nl), rng.uniform(0, 2 * math.pi, nl)
    lay = [dict(nx=n, ny=n, dx=dx, ox=-n / 2 * dx, oy=-n / 2 * dx, ht=HT[i], vx=float(v[i] * np.cos(a[i])),
                vy=float(v[i] * np.sin(a[i])), alpha=1.0) for i in range(nl)]
    return lay, wt, int(rng.integers(20, 4000))


def _screens(c, wt, seed):
    """Von Karman phase screens (metres of path), FP64 on the device."""
    n, dx = c["nx"], c["sdx"]
    g = torch.Generator(device=DEV).manual_seed(seed)
    f = torch.fft.fftfreq(n, dx, dtype=torch.float64, device=DEV)
    amp = (f[:, None] ** 2 + f[None, :] ** 2 + L0 ** -2) ** (-11.0 / 12)
    amp *= math.sqrt(0.0229 * R0 ** (-5 / 3)) * 0.5e-6 / (2 * math.pi) / (n * dx)
    amp[0, 0] = 0
    out = []
    for i in range(0, len(wt), 2):
        z = torch.complex(torch.randn(n, n, dtype=torch.float64, device=DEV, generator=g),
                          torch.randn(n, n, dtype=torch.float64, device=DEV, generator=g))
        z = torch.fft.fft2(z.mul_(amp))
        out.append(z.real * math.sqrt(wt[i]))
        if i + 1 < len(wt):
            out.append(z.imag * math.sqrt(wt[i + 1]))
    return out


def _mirrors(D, seed):
    """Two mirror grids (ground and 9 km) at 0.5 m pitch that cover every footprint."""
    rng = np.random.default_rng(seed + 77)
    grids, surf = [], []
    for ht, n in ((0.0, int(D / 0.5) + 9), (9000.0, int(D / 0.5) + 17)):
        o = -(n // 2) * 0.5
        x = o + 0.5 * np.arange(n)
        X, Y = np.meshgrid(x, x)
        s = np.zeros((n, n))
        for _ in range(6):
            kx, ky = rng.uniform(-1.2, 1.2, 2)
            s += rng.normal(0, 1.5e-7) * np.cos(kx * X + ky * Y + rng.uniform(0, 2 * np.pi))
        grids.append(dict(nx=n, ny=n, dx=0.5, ox=o, oy=o, ht=ht, alpha=-1.0))
        surf.append(s)
    return grids, surf


def _terms(cfg, nwfs, seed):
    """Tip/tilt, focus and uplink tip/tilt of every sensor in closed loop."""
    rng = np.random.default_rng(seed + 78)
    llt = bool(cfg["has_llt"])
    return [dict(ptt=(0.0, float(rng.normal(0, 1e-7)), float(rng.normal(0, 1e-7))), focus_tel=float(rng.normal(0, 2e-9)),
                 focus_llt=float(rng.normal(0, 1e-9)) if llt else 0.0,
                 lltptt=(float(rng.normal(0, 1e-7)), float(rng.normal(0, 1e-7))) if llt else (0.0, 0.0))
            for _ in range(nwfs)]


def _phase(c, cfg, s, seed):
    """Phase of one sensor's subapertures (and its laser pupil) as the caller of an imaging call holds it."""
    lay, wt, isim = _layers(c, seed)
    scr = _screens(c, wt, seed)
    opd = _trace(cfg, s, 0, lay, scr, isim).float().reshape(-1)
    llt = _trace_llt(cfg, s, 0, lay, scr, isim).float().reshape(-1) if cfg["has_llt"] else None
    return opd, llt


def _detector(c, seed):
    """Spot intensities of the case's mean, and the camera's noise parameters."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    x = torch.rand(c["n"], device=DEV, generator=g)
    return (x * x * x) * (4 * c["mean"])


class _State:
    pass


def prepare(case, seed):
    c = case
    st = _State()
    st.case = c
    ctx = st.ctx = shwfs.Context(0)
    kind = c["kind"]
    if kind == "noise":
        st.x0 = _detector(c, seed)
        st.x = torch.empty_like(st.x0)
        st.seed = seed
        st.stream = torch.cuda.ExternalStream(ctx.stream)
        torch.cuda.synchronize()
        return st
    ctx.set_dt(DT)
    if kind == "science":
        lay, wt, st.isim = _layers(c, seed)
        ctx.atm_set(lay, [t.cpu().numpy() for t in _screens(c, wt, seed)])
        x, y, a = _aperture(c["D"], c["sdx"])
        ctx.evl_set_aper(x, y, c["sdx"], a)
        for d in _dirs(c):
            ctx.evl_add_dir(*d)
        w = c["wvls"]
        ctx.evl_set_psf(_wvls(c), [c["nembed"]] * w, [c["psfsize"]] * w, pttr=c["pttr"])
        return st
    ctx.set_form(shwfs.SHWFS_FORM_TC if c["form"] == "tc" else shwfs.SHWFS_FORM_FFT)
    st.nwfs, n = 0, 0
    for cfg in _members(c):
        s = _setup(cfg)
        if kind == "geom":
            ip = ctx.powfs_add(nsa=s.nsa, nopd=s.nopd, embfac=1, notf=0, pixpsax=0, pixpsay=0, dsa=cfg["dsa"], dx=s.dx,
                               hs=cfg["hs"], areascale=1.0, wvl=cfg["wvl"], gradtype=shwfs.SHWFS_GRAD_ZTILT)
            ctx.powfs_set_geom(ip, s.get("origx"), s.get("origy"), s.get("amp"))
        else:
            ip = s.load(ctx)
        for k in range(cfg["nwfs"]):
            i = ctx.wfs_add(ipowfs=ip, thetax=cfg["thetax"][k], thetay=cfg["thetay"][k], hs=cfg["hs"], hc=0.0,
                            misregx=0.0, misregy=0.0, sigsim=cfg["siglev"], wvlwt=1.0, noisy=0)
            if kind != "geom":
                s.load_wfs(ctx, i)
            st.nwfs += 1
            n += 2 * s.nsa
    if kind == "images":
        cfg = _config(c)
        s = _setup(cfg)
        st.opd, st.llt = _phase(c, cfg, s, seed)
        st.ints = torch.empty(s.nsa * s.npix, device=DEV)
        st.grad = torch.zeros(2 * s.nsa, device=DEV)
        torch.cuda.synchronize()
        return st
    lay, wt, st.isim = _layers(c, seed)
    ctx.atm_set(lay, [t.cpu().numpy() for t in _screens(c, wt, seed)])
    st.out = np.zeros(n)
    if kind == "loop":
        st.grids, st.surf = _mirrors(c["D"], seed)
        st.terms = _terms(_config(c), st.nwfs, seed)
    return st


def run(state):
    st, ctx, kind = state, state.ctx, state.case["kind"]
    if kind == "noise":
        c = st.case
        with torch.cuda.stream(st.stream):  # the frame's intensities, then the camera's noise on them
            st.x.copy_(st.x0)
        ctx.addnoise_dev(st.x, seed=st.seed, stream=1, frame=3, bkgrnd=c["bkgrnd"], bkgrndc=c["bkgrnd"], rne=c["rne"])
        return st.x
    if kind == "science":
        c = st.case
        ctx.evl_psf_reset()
        wfe = []
        for f in range(c["frames"]):
            ctx.evl_queue(st.isim + f, do_psf=True)
            wfe.append(ctx.evl_sync())
        psf = [ctx.evl_psf(e, w)[0] for e in range(c["dirs"]) for w in range(c["wvls"])]
        return dict(wfe=np.stack([w for w, _ in wfe]), coeff=np.stack([q for _, q in wfe]), psf=np.stack(psf))
    if kind == "images":
        ctx.ints_grad_dev(0, 0, st.opd, st.llt, st.ints, st.grad)
        return dict(ints=st.ints, grad=st.grad)
    if kind == "loop":
        ctx.dm_set(st.grids, st.surf)
        for i, t in enumerate(st.terms):
            ctx.wfs_set_opd_terms(i, use_dm=True, **t)
    if kind == "batch":
        ctx.frame_graph(st.isim, 0, st.nwfs)
    else:
        ctx.frame_queue(st.isim, 0, st.nwfs)
    return ctx.frame_sync_range(0, st.nwfs, out=st.out)


# ---------------------------------------------------------------------------
# the work of a pass
# ---------------------------------------------------------------------------
def work(case):
    c = case
    if c["kind"] == "noise":
        return dict(bytes=8 * c["n"], flops=100 * c["n"])
    foot = min(c["nx"], c["D"] / c["sdx"] + 2) ** 2 * 4 * c["layers"]  # screen points under the pupils, once
    if c["kind"] == "science":
        npt = math.pi / 4 * (1 - 0.12 ** 2) * (c["D"] / c["sdx"]) ** 2
        N, ps = c["nembed"], c["psfsize"]
        per = c["dirs"] * (npt * (13 * c["layers"] + 16) + c["wvls"] * (
            (c["D"] / c["sdx"] + ps) * 5 * N * math.log2(N) + 14 * npt))
        return dict(bytes=c["frames"] * (foot + 4 * npt) + c["dirs"] * c["wvls"] * ps * ps * 4, flops=c["frames"] * per)
    byt = 0 if c["kind"] == "images" else foot
    flops = 0
    for cfg in _members(c):
        nsa = max(1, math.pi / 4 * (1 - 0.12 ** 2) * cfg["order"] ** 2)
        no, N, npix, nw = cfg["notf"] // cfg["embfac"], cfg["notf"], cfg["pixpsa"] ** 2, cfg["nwfs"]
        byt += nsa * no * no * 4 + nw * nsa * 8
        if c["kind"] == "images":
            byt += nsa * (no * no + npix) * 4
        else:
            flops += nw * nsa * no * no * 13 * (c["layers"] + (2 if c["kind"] == "loop" else 0))
        if c["kind"] == "geom":
            flops += nw * nsa * no * no * 12
            continue
        byt += (nsa * N * N * 8 if cfg["has_llt"] else N * N * 4) + (nw * nsa * npix * 8 if cfg["phytype"] == 1 else 0)
        flops += nw * nsa * (15 * N * N * math.log2(N * N) + 20 * N * N)
    return dict(bytes=byt, flops=flops)


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def _t(a):
    return torch.as_tensor(np.asarray(a), device=DEV)


def _bilinear(scr, jx, jy, wx, wy, wrap):
    """scr[jy, jx] interpolated at every (row, column) of each block; jx, wx (nsa, nx), jy, wy (nsa, ny)."""
    n1, n0 = scr.shape
    if wrap:
        jx, jy = jx % n0, jy % n1
        kx, ky = (jx + 1) % n0, (jy + 1) % n1
        ok = None
    else:
        ok = ((jy >= 0) & (jy < n1 - 1))[:, :, None] & ((jx >= 0) & (jx < n0 - 1))[:, None, :]
        jx, jy = jx.clamp(0, n0 - 2), jy.clamp(0, n1 - 2)
        kx, ky = jx + 1, jy + 1
    wx, wy = wx[:, None, :], wy[:, :, None]
    at = lambda y, x: scr[y[:, :, None], x[:, None, :]]  # noqa: E731
    v = (at(jy, jx) * (1 - wx) + at(jy, kx) * wx) * (1 - wy) + (at(ky, jx) * (1 - wx) + at(ky, kx) * wx) * wy
    return v if ok is None else torch.where(ok, v, torch.zeros_like(v))


def _trace_grid(ox, oy, nopd, dx, theta, hs, shift, lay, scr, isim, mir=()):
    """OPD (nsa, nopd, nopd) of a pupil: the layers with wind and wrap, then the mirrors without."""
    i = torch.arange(nopd, dtype=torch.float64, device=DEV) * dx
    X, Y = ox[:, None] + i, oy[:, None] + i
    acc = torch.zeros(len(ox), nopd, nopd, dtype=torch.float64, device=DEV)
    for l, s, wrap in [(l, s, True) for l, s in zip(lay, scr)] + [(l, s, False) for l, s in mir]:
        scale = 1 - l["ht"] / hs if math.isfinite(hs) else 1.0
        mx = l["ht"] * theta[0] + (shift[0] - l["vx"] * DT * isim if wrap else 0.0)
        my = l["ht"] * theta[1] + (shift[1] - l["vy"] * DT * isim if wrap else 0.0)
        x, y = (X * scale + mx - l["ox"]) / l["dx"], (Y * scale + my - l["oy"]) / l["dx"]
        jx, jy = torch.floor(x), torch.floor(y)
        acc += l["alpha"] * _bilinear(s, jx.long(), jy.long(), x - jx, y - jy, wrap)
    return acc


def _trace(cfg, s, k, lay, scr, isim, mir=()):
    return _trace_grid(_t(s.get("origx")), _t(s.get("origy")), s.nopd, s.dx, (cfg["thetax"][k], cfg["thetay"][k]), cfg["hs"],
                       (0.0, 0.0), lay, scr, isim, mir)


def _trace_llt(cfg, s, k, lay, scr, isim):
    ox, oy = cfg["llt_ox"], cfg["llt_oy"]
    o = torch.full((1,), (1 - s.llt_nx) * s.dx / 2, dtype=torch.float64, device=DEV)
    return _trace_grid(o, o, s.llt_nx, s.dx, (cfg["thetax"][k] - ox / cfg["hs"], cfg["thetay"][k] - oy / cfg["hs"]),
                       cfg["hs"], (ox, oy), lay, scr, isim)


def _points(s):
    """Pupil coordinates of every OPD point, (nsa, ny, nx)."""
    i = torch.arange(s.nopd, dtype=torch.float64, device=DEV) * s.dx
    x = (_t(s.get("origx"))[:, None, None] + i[None, None, :]).expand(-1, s.nopd, -1)
    y = (_t(s.get("origy"))[:, None, None] + i[None, :, None]).expand(-1, -1, s.nopd)
    return x, y


def _psf(opd, amp, wvl, N):
    """|FFT|^2 of the padded field."""
    return torch.fft.fft2(amp * torch.exp(2j * math.pi / wvl * opd), s=(N, N)).abs() ** 2


def _images(cfg, s, opd, llt):
    """Noise-free pixel intensities (nsa, npix)."""
    N, nsa = s.notf, s.nsa
    amp = _t(s.get("amp")).reshape(nsa, s.nopd, s.nopd)
    up = 1.0
    if llt is not None:
        n = s.llt_nx
        up = torch.fft.fft2(_psf(llt, _t(s.get("lltamp")).reshape(n, n), cfg["wvl"], N) / (n * cfg["embfac"]) ** 2).conj()
    idx, wt = _t(s.simap_idx()).long(), _t(s.get("simap_wt")).reshape(-1, 4)
    idx = idx.reshape(-1, 4)
    wt = torch.where(idx >= 0, wt, torch.zeros_like(wt))
    tf = _t(s.get("etf")).reshape(nsa, N, N) if cfg["has_llt"] else _t(s.get("nominal")).reshape(1, N, N)
    nw = s.nopd * cfg["embfac"]
    norm = cfg["siglev"] * s.areascale / (s.nopd * nw) ** 2
    out = []
    for a in range(0, nsa, 512):
        otf = torch.fft.fft2(_psf(opd[a:a + 512], amp[a:a + 512], cfg["wvl"], N)) * up
        img = torch.fft.ifft2(otf * (tf[a:a + 512] if cfg["has_llt"] else tf)).real.reshape(-1, N * N)
        out.append((img[:, idx.clamp(min=0)] * wt).sum(-1) * norm)
    return torch.cat(out)


def _gradients(cfg, s, ints):
    """Matched-filter or centre-of-gravity gradients (2 nsa)."""
    n = s.npix
    if cfg["phytype"] == 1:
        m = _t(s.get("mtche")).reshape(s.nsa, n, 2)
        scale = _t(s.get("i0sum")) / ints.sum(1)
        scale = torch.where((scale > 0) & (scale <= 10), scale, torch.ones_like(scale))
        g = (m * ints[:, :, None]).sum(1) * scale[:, None]
        return torch.cat([g[:, 0], g[:, 1]])
    p = torch.arange(n, device=DEV)
    v = torch.where(ints > 0, ints, torch.zeros_like(ints))
    c = (s.cfg["pixpsa"] - 1) / 2
    gx = ((v * (p % s.cfg["pixpsa"])).sum(1) / v.sum(1) - c) * cfg["pixtheta"]
    gy = ((v * (p // s.cfg["pixpsa"])).sum(1) / v.sum(1) - c) * cfg["pixtheta"]
    return torch.cat([gx, gy])


def _ztilt(s, opd):
    """Amplitude-weighted least-squares plane of every subaperture (2 nsa)."""
    x, y = _points(s)
    x0, y0 = x.mean((1, 2), keepdim=True), y.mean((1, 2), keepdim=True)
    a = _t(s.get("amp")).reshape(opd.shape)
    b = torch.stack([torch.ones_like(x), x - x0, y - y0]).flatten(2)  # 3, nsa, points
    A = torch.einsum("isp,jsp,sp->sij", b, b, a.flatten(1))
    r = torch.einsum("isp,sp,sp->si", b, a.flatten(1), opd.flatten(1))
    g = torch.linalg.solve(A, r)
    return torch.cat([g[:, 1], g[:, 2]])


@functools.lru_cache(maxsize=None)
def _aperture(D, dx):
    return aperture(D, 0.12 * D, dx)


def _dirs(c):
    n = c["dirs"]
    return [(15 * AS2RAD * math.cos(2 * math.pi * k / n) * (k > 0), 15 * AS2RAD * math.sin(2 * math.pi * k / n), math.inf)
            for k in range(n)]


def _wvls(c):
    return [1.25e-6, 1.65e-6, 2.2e-6][:c["wvls"]]


def _exact_science(c, seed):
    lay, wt, isim = _layers(c, seed)
    scr = _screens(c, wt, seed)
    x, y, a = (_t(v) for v in _aperture(c["D"], c["sdx"]))
    dx, N, h = c["sdx"], c["nembed"], c["psfsize"] // 2
    X, Y = torch.round((x - x.min()) / dx).long(), torch.round((y - y.min()) / dx).long()
    nX, nY = int(X.max()) + 1, int(Y.max()) + 1
    i = torch.arange(max(nX, nY), dtype=torch.float64, device=DEV) * dx
    B = torch.stack([torch.ones_like(x), x, y])
    mcc = (B * a) @ B.T
    keep = torch.cat([torch.arange(N - h, N), torch.arange(0, h)]).to(DEV)  # the centre of the shifted image
    wfe, coeff, psf = [], [], torch.zeros(c["dirs"], c["wvls"], 2 * h, 2 * h, dtype=torch.float64, device=DEV)
    for f in range(c["frames"]):
        rows = []
        for e, (tx, ty, _) in enumerate(_dirs(c)):
            o = torch.zeros(nY, nX, dtype=torch.float64, device=DEV)
            for l, s in zip(lay, scr):
                u = (x.min() + i[:nX] + l["ht"] * tx - l["vx"] * DT * (isim + f) - l["ox"]) / l["dx"]
                v = (y.min() + i[:nY] + l["ht"] * ty - l["vy"] * DT * (isim + f) - l["oy"]) / l["dx"]
                ju, jv = torch.floor(u), torch.floor(v)
                o += _bilinear(s, ju.long()[None], jv.long()[None], (u - ju)[None], (v - jv)[None], True)[0]
            p = o[Y, X]
            b = (B * a) @ p
            cf = torch.linalg.solve(mcc, b)
            tot, pis, ptt = (a * p * p).sum(), b[0] ** 2 / mcc[0, 0], (b * cf).sum()
            rows.append((torch.stack([tot - pis, ptt - pis, tot - ptt]), cf))
            if c["pttr"]:
                p = p - cf @ B
            for w, wvl in enumerate(_wvls(c)):
                E = torch.zeros(nX, nY, dtype=torch.complex128, device=DEV)
                E[X, Y] = a * torch.exp(2j * math.pi / wvl * p)
                F = torch.fft.fft(torch.fft.fft(E, n=N, dim=0)[keep], n=N, dim=1)[:, keep]
                psf[e, w] += F.abs() ** 2
        wfe.append(torch.stack([r[0] for r in rows]))
        coeff.append(torch.stack([r[1] for r in rows]))
    num = lambda t: t.cpu().numpy()  # noqa: E731
    return dict(wfe=num(torch.stack(wfe)), coeff=num(torch.stack(coeff)), psf=num(psf.reshape(-1, 2 * h, 2 * h)))


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "noise":
        return None
    if kind == "science":
        return _exact_science(c, seed)
    if kind == "images":
        cfg = _config(c)
        s = _setup(cfg)
        opd, llt = _phase(c, cfg, s, seed)
        opd = opd.double().reshape(s.nsa, s.nopd, s.nopd)
        ints = _images(cfg, s, opd, None if llt is None else llt.double().reshape(s.llt_nx, s.llt_nx))
        return dict(ints=ints.reshape(-1).cpu().numpy(), grad=_gradients(cfg, s, ints).cpu().numpy())
    lay, wt, isim = _layers(c, seed)
    scr = _screens(c, wt, seed)
    out = []
    for cfg in _members(c):
        s = _setup(cfg)
        mir, terms = (), None
        if kind == "loop":
            grids, surf = _mirrors(c["D"], seed)
            mir = [(g, _t(v)) for g, v in zip(grids, surf)]
            terms = _terms(cfg, cfg["nwfs"], seed)
        for k in range(cfg["nwfs"]):
            opd = _trace(cfg, s, k, lay, scr, isim, mir)
            llt = _trace_llt(cfg, s, k, lay, scr, isim)[0] if cfg["has_llt"] and kind != "geom" else None
            if terms:
                t = terms[k]
                x, y = _points(s)
                r = x * x + y * y
                opd = opd + t["ptt"][0] + t["ptt"][1] * x + t["ptt"][2] * y + t["focus_tel"] * (r - r.mean())
                if llt is not None:
                    r = (x - cfg["llt_ox"]) ** 2 + (y - cfg["llt_oy"]) ** 2
                    opd = opd + t["focus_llt"] * (r - r.mean())
                    i = (torch.arange(s.llt_nx, dtype=torch.float64, device=DEV) - (s.llt_nx - 1) / 2) * s.dx
                    llt = llt + t["lltptt"][0] * i[None, :] + t["lltptt"][1] * i[:, None]
            out.append(_ztilt(s, opd) if kind == "geom" else _gradients(cfg, s, _images(cfg, s, opd, llt)))
    return torch.cat(out).cpu().numpy()
