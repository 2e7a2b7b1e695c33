"""Imaging at FFT 64, 128 and 256 and the cropped science PSF against plain
FP64 transforms.

FFT 64 (ints_n64_kernel): pupils of 16, 32 and 64 points (the fixed size and
the general one), a DTF nominal or an ETF with an uplink OTF (which the FFT
passes form at 64 points), and pixel counts below, at and above a block's
threads.  FFT 128 and 256 (the FFT passes): pupils that fill their last tile of
columns and pupils that do not.  Spots are compact, lopsided and off centre, the
transfer functions as wide as the spots, and the pixels lie around the spots.
Tolerance of a noise-free intensity, relative to the subaperture's largest: the
rounding of three two-dimensional transforms is white, 3 log2(N^2) 2^-24 <= 48 *
2^-24 of the image's 2-norm, and the 2-norm is at most N of its largest pixel, so
2.9e-6 rms a pixel; four times that for the largest of 256.  A centre of
gravity moves by the pixels' errors over their sum.  Images that are transposed,
mirrored, uniform or lack a transfer function are off by a hundred times the
tolerance and more (checked on the reference).

Science PSF: crops of at most 256 pixels run the two-pass transforms
(evl_fold_rows_kernel) for rows of 512 to 4096 points, larger crops the full
ones; columns run the two passes (evl_fold_cols_kernel) in launches of more
lines than the chip holds blocks of the full transforms; apertures of odd and
even width; PSFs read whole and in parts.  Tolerance: within 2e-5 of the peak,
as the science path's reference test."""
import math

import numpy as np
import pytest

from tests.conftest import cuda_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")]


TOL = 1.2e-5


def _tf(N, wide):
    """Transfer function of a lopsided kernel: a blob off the origin and a smaller one beside it."""
    i = np.fft.fftfreq(N, 1 / N)
    y, x = i[:, None], i[None]
    k = np.exp(-((x - wide) / (1.2 * wide)) ** 2 - ((y + 0.6 * wide) / (0.7 * wide)) ** 2)
    k += 0.4 * np.exp(-((x + 0.8 * wide) ** 2 + (y - 1.1 * wide) ** 2) / (0.6 * wide) ** 2)
    return np.fft.fft2(k / k.sum())


def _phase(rng, n, nopd):
    """Tilt, coma and a little noise, in waves."""
    u = (np.arange(nopd) + 0.5) / nopd * 2 - 1
    y, x = u[:, None], u[None]
    t = rng.uniform(0.15, 0.4, (n, 4, 1, 1))
    return t[:, 0] * x - t[:, 1] * y + (t[:, 2] * x + 0.5 * t[:, 3] * y) * (x * x + y * y) + rng.normal(0, 0.01, (n, nopd, nopd))


def _psf(a, phase, N):
    return np.abs(np.fft.fft2(a * np.exp(2j * np.pi * phase), s=(N, N))) ** 2


@pytest.mark.parametrize("N,nopd,pix", [(64, 32, 5), (64, 32, 12), (64, 32, 16), (64, 16, 8), (64, 64, 11),
                                        (128, 64, 16), (128, 8, 7), (256, 128, 9), (256, 4, 16)])
@pytest.mark.parametrize("lgs", [False, True])
def test_images_match_plain(N, nopd, pix, lgs):
    import torch
    from maos_b200 import shwfs
    rng = np.random.default_rng(nopd * 100 + pix)
    nsa, nllt, wvl, pixt = 5, nopd, 0.6e-6, 1e-6  # an LLT pupil has the subapertures' sampling
    npix, wide = pix * pix, max(1.5, 0.5 * N / nopd)
    amp = rng.uniform(0.5, 1, (nsa, nopd, nopd))
    amp /= np.sqrt((amp ** 2).sum((1, 2), keepdims=True))
    lltamp = rng.uniform(0.5, 1, (nllt, nllt))
    lltamp /= np.sqrt((lltamp ** 2).sum())
    opd = (wvl * _phase(rng, nsa, nopd)).astype(np.float32)
    llt = (wvl * _phase(rng, 1, nllt)[0]).astype(np.float32)
    f = np.fft.fftfreq(N)
    if lgs:
        tf = np.stack([_tf(N, wide * s) for s in np.linspace(0.8, 1.2, nsa)])
    else:  # real and even, as the transform of a centred pixel
        tf = np.exp(-(3 * wide * f[:, None]) ** 2 - (6 * wide * f[None]) ** 2)[None]
    # the reference: images (row y, column x), then pixels of four weighted taps around the mean spot
    field = opd.astype(float) / wvl
    otf = np.fft.fft2(_psf(amp, field, N))
    up = np.conj(np.fft.fft2(_psf(lltamp, llt.astype(float) / wvl, N) / N ** 2)) if lgs else 1.0
    image = lambda o: np.fft.ifft2(o).real * 700.0 / (nopd * N) ** 2  # noqa: E731
    img = image(otf * up * tf)
    cy, cx = np.unravel_index(img.mean(0).argmax(), (N, N))
    step = max(1, int(round(3 * wide * 2 / pix)))
    py, px = np.meshgrid(cy + (np.arange(pix) - pix // 2) * step, cx + (np.arange(pix) - pix // 2) * step, indexing="ij")
    idx = np.stack([(py + a) % N * N + (px + b) % N for a in (0, 1) for b in (0, 1)], -1).reshape(npix, 4)
    idx[rng.uniform(size=idx.shape) < 0.2] = -1
    idx[:, 0] = (py % N * N + px % N).ravel()
    wt = rng.uniform(0.2, 1, (npix, 4))
    pixels = lambda m: (np.where(idx >= 0, m.reshape(nsa, -1)[:, np.maximum(idx, 0)], 0) * wt).sum(-1)  # noqa: E731
    ref = pixels(img)
    peak = ref.max(1, keepdims=True)
    wrong = [img.transpose(0, 2, 1), image(otf * up), np.roll(img[:, ::-1], 1, 1), np.roll(img[:, :, ::-1], 1, 2),
             np.full_like(img, img.mean())] + ([image(otf * tf), image(otf * np.conj(up) * tf)] if lgs else [])
    for m in wrong:
        assert (np.abs(pixels(m) - ref) / peak).max(1).min() > 100 * TOL

    ctx = shwfs.Context(0)
    ip = ctx.powfs_add(nsa=nsa, nopd=nopd, embfac=N // nopd, notf=N, pixpsax=pix, pixpsay=pix, pixthetax=pixt,
                       pixthetay=pixt, wvl=wvl, dsa=0.5, dx=0.5 / nopd, areascale=1.0, hs=90e3 if lgs else math.inf,
                       has_etf=int(lgs), has_llt=int(lgs), llt_nx=nllt if lgs else 0, gradtype=shwfs.SHWFS_GRAD_COG,
                       sigmatch=1)
    ctx.powfs_set_geom(ip, np.zeros(nsa), np.zeros(nsa), amp, np.ones(nsa))
    ctx.powfs_set_simap(ip, idx, wt)
    if lgs:
        ctx.powfs_set_etf(ip, tf.reshape(nsa, -1))
        ctx.powfs_set_lltamp(ip, lltamp)
    else:
        ctx.powfs_set_nominal(ip, tf)
    iw = ctx.wfs_add(ipowfs=ip, thetax=0.0, thetay=0.0, hs=90e3 if lgs else math.inf, hc=0.0, misregx=0.0, misregy=0.0,
                     sigsim=700.0, wvlwt=1.0, noisy=0)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    ints, grad = torch.full((nsa * npix,), -1.0, device="cuda"), torch.zeros(2 * nsa, device="cuda")
    d_opd, d_llt = dev(opd), dev(llt)
    torch.cuda.synchronize()
    ctx.ints_grad_dev(iw, 0, d_opd, d_llt if lgs else None, ints, grad)
    ctx.sync()
    ctx.close()
    got = ints.double().cpu().numpy().reshape(nsa, npix)
    assert (np.abs(got - ref) / peak).max() <= TOL
    p = np.arange(npix)
    v = np.where(ref > 0, ref, 0)
    cog = np.stack([(v * (q - (pix - 1) / 2)).sum(1) / v.sum(1) for q in (p % pix, p // pix)]) * pixt
    off = npix * pix * TOL * peak[:, 0] / v.sum(1) * pixt
    assert (np.abs(grad.double().cpu().numpy().reshape(2, nsa) - cog) <= off).all()


@pytest.mark.parametrize("N,ps,nx,nevl", [
    (512, 256, 301, 1), (512, 258, 301, 1), (2048, 1100, 301, 1), (1024, 50, 1024, 1), (2048, 256, 130, 1), (4096, 16, 701, 1), (4096, 256, 700, 1),
    (512, 256, 301, 3), (1024, 50, 1024, 12), (2048, 256, 130, 3), (4096, 16, 701, 19), (4096, 256, 700, 2)])
@pytest.mark.parametrize("pttr", [0, 1])
def test_cropped_psf_matches_plain(N, ps, nx, nevl, pttr):
    from maos_b200 import shwfs
    rng = np.random.default_rng(N + ps)
    dx, wvl, nxs, sdx = 1 / 32, 1.5e-6, 256, 0.25
    ix, iy = np.meshgrid(np.arange(nx), np.arange(nx - 7))
    keep = (ix - nx / 2) ** 2 + (iy - nx / 2) ** 2 <= (nx / 2) ** 2
    keep[0, 0] = keep[-1, -1] = keep[0, -1] = True  # the whole bounding box
    ix, iy = ix[keep], iy[keep]
    x, y = (ix - nx / 2) * dx, (iy - nx / 2) * dx
    amp = rng.uniform(0.5, 1, len(x))
    amp /= amp.sum()
    ctx = shwfs.Context(0)
    ctx.set_dt(1 / 800)
    t = np.arange(nxs) * 2 * np.pi / nxs
    scr = 2e-7 * (np.cos(3 * t)[None] + np.sin(2 * t)[:, None] + np.cos(7 * t[None] + 5 * t[:, None]))
    ctx.atm_set([dict(nx=nxs, ny=nxs, dx=sdx, ox=-nxs / 2 * sdx, oy=-nxs / 2 * sdx, ht=0.0, vx=0.0, vy=0.0, alpha=1.0)], [scr])
    ctx.evl_set_aper(x, y, dx, amp)
    for _ in range(nevl):
        ctx.evl_add_dir(0.0, 0.0)
    ctx.evl_set_psf([wvl], [N], [ps], pttr=pttr)
    ctx.evl_queue(0, do_psf=True)
    wfe, coeff = ctx.evl_sync()
    got, n = zip(*(ctx.evl_psf(e, 0) for e in range(nevl)))
    assert set(n) == {1}
    u, v = x / sdx + nxs / 2, y / sdx + nxs / 2
    ju, jv = np.floor(u).astype(int), np.floor(v).astype(int)
    wu, wv = u - ju, v - jv
    at = lambda a, b: scr[a % nxs, b % nxs]  # noqa: E731
    o = (at(jv, ju) * (1 - wu) + at(jv, ju + 1) * wu) * (1 - wv) + (at(jv + 1, ju) * (1 - wu) + at(jv + 1, ju + 1) * wu) * wv
    B = np.stack([np.ones_like(x), x, y])
    c = np.linalg.solve((B * amp) @ B.T, (B * amp) @ o)
    assert np.allclose(coeff[0], c, rtol=0, atol=1e-4 * np.abs(c).max())
    if pttr:
        o = o - c @ B
    E = np.zeros((nx, nx - 7), complex)
    E[ix, iy] = amp * np.exp(2j * np.pi / wvl * o)
    h = ps // 2
    f = np.concatenate([np.arange(N - h, N), np.arange(h)])
    F = np.fft.fft(np.fft.fft(E, n=N, axis=0)[f], n=N, axis=1)[:, f]
    ref = np.abs(F) ** 2
    assert np.abs(np.stack(got) - ref).max() <= 2e-5 * ref.max()
    ctx.close()


def test_first_psf_read_allocates_nothing():
    import torch
    from maos_b200 import shwfs

    def exposure(ps):
        ctx = shwfs.Context(0)
        x, y = (a.ravel() / 16.0 for a in np.meshgrid(np.arange(64), np.arange(64)))
        ctx.evl_set_aper(x, y, 1 / 16, np.ones(64 * 64))
        ctx.evl_add_dir(0.0, 0.0)
        ctx.evl_set_psf([1e-6], [1024], [ps])
        ctx.evl_queue(0, do_psf=True)
        ctx.evl_sync()
        before = torch.cuda.mem_get_info()[0]
        ctx.evl_psf(0, 0)
        return ctx, before, torch.cuda.mem_get_info()[0]

    ctx, _, _ = exposure(16)  # loads the read's kernel
    ctx.close()
    ctx, before, after = exposure(1024)
    ctx.close()
    assert after == before
