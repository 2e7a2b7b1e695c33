"""Ray trace of 16x16 and 32x32 pupils (geom_rows_kernel) against a plain FP64
bilinear trace: launches of few and of many pupils (two and eight rows per
lane), footprints that cross a screen edge, and pupil sampling finer than,
equal to and coarser than the screen's (rows that reuse, advance by or skip a
screen row), with and without mirror grids.

Tolerance: a layer's value is off by the FP32 rounding of the screen, of the
point's FP32 coordinate within its line (at most 64 steps: 64 * 2^-23 of a
cell, times the difference of two neighbours) and of five operations:
(1 + 2*64 + 5) * 2^-23 = 1.6e-5 of the largest screen value, per layer."""
import numpy as np
import pytest

from tests.conftest import cuda_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")]


def _plain(ox, oy, nopd, dx, layers, screens, wrap):
    i = np.arange(nopd) * dx
    out = np.zeros((len(ox), nopd, nopd))
    for l, s in zip(layers, screens):
        ny, nx = s.shape
        x, y = (ox[:, None] + i - l["ox"]) / l["dx"], (oy[:, None] + i - l["oy"]) / l["dx"]
        jx, jy = np.floor(x).astype(int), np.floor(y).astype(int)
        wx, wy = (x - jx)[:, None, :], (y - jy)[:, :, None]
        ok = np.ones((len(ox), nopd, nopd), bool)
        if not wrap:
            ok = ((jx >= 0) & (jx < nx - 1))[:, None, :] & ((jy >= 0) & (jy < ny - 1))[:, :, None]
        at = lambda a, b: s[(a % ny)[:, :, None], (b % nx)[:, None, :]]  # noqa: E731
        v = (at(jy, jx) * (1 - wx) + at(jy, jx + 1) * wx) * (1 - wy) + (
            at(jy + 1, jx) * (1 - wx) + at(jy + 1, jx + 1) * wx) * wy
        out += l["alpha"] * np.where(ok, v, 0.0)
    return out


@pytest.mark.parametrize("mirror", [False, True])
@pytest.mark.parametrize("step", [0.07, 0.83, 1.0, 1.9])
@pytest.mark.parametrize("nopd,nsa", [(16, 3), (16, 1601), (32, 3), (32, 401)])
def test_rows_trace_matches_plain(nopd, nsa, step, mirror):
    import torch
    from maos_b200 import shwfs
    rng = np.random.default_rng(nopd + nsa)
    sdx, nx, ny = 1.0 / 32, 96, 160
    dx = step * sdx
    ox, oy = rng.uniform(-3.5, 3.5, nsa), rng.uniform(-4.5, 4.5, nsa)  # beyond the screen edges too
    layers = [dict(nx=nx, ny=ny, dx=sdx, ox=-1.5, oy=-2.5, ht=0.0, vx=0.0, vy=0.0, alpha=a) for a in (1.0, -0.4, 2.0)]
    screens = [rng.standard_normal((ny, nx)) for _ in layers]
    ctx = shwfs.Context(0)
    ip = ctx.powfs_add(nsa=nsa, nopd=nopd, embfac=1, notf=0, pixpsax=0, pixpsay=0, dsa=nopd * dx, dx=dx, hs=np.inf,
                       areascale=1.0, wvl=1e-6, gradtype=shwfs.SHWFS_GRAD_ZTILT)
    ctx.powfs_set_geom(ip, ox, oy, np.ones(nsa * nopd * nopd))
    iw = ctx.wfs_add(ipowfs=ip, thetax=0.0, thetay=0.0, hs=np.inf, hc=0.0, misregx=0.0, misregy=0.0, sigsim=1.0,
                     wvlwt=1.0, noisy=0)
    ctx.atm_set(layers, screens)
    ref = _plain(ox, oy, nopd, dx, layers, screens, True)
    peak = sum(abs(l["alpha"]) * np.abs(s).max() for l, s in zip(layers, screens))
    if mirror:  # a coarse grid that some points leave
        grid = dict(nx=24, ny=20, dx=0.3, ox=-3.1, oy=-2.9, ht=0.0, alpha=-1.0)
        surf = rng.standard_normal((20, 24))
        ctx.dm_set([grid], [surf])
        ctx.wfs_set_opd_terms(iw, use_dm=True)
        ref += _plain(ox, oy, nopd, dx, [grid], [surf], False)
        peak += np.abs(surf).max()
    opd = torch.full((nsa * nopd * nopd,), 7.0, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    ctx.raytrace_dev(iw, 0, opd)
    ctx.sync()
    o = opd.double().cpu().numpy().reshape(ref.shape)
    d = np.abs(o - ref)
    if mirror:  # a point within a coordinate's rounding of the grid's edge may fall on either side of it
        x = (ox[:, None] + np.arange(nopd) * dx - grid["ox"]) / grid["dx"]
        y = (oy[:, None] + np.arange(nopd) * dx - grid["oy"]) / grid["dx"]
        near = lambda v, n: (np.abs(v) < 1e-5) | (np.abs(v - (n - 1)) < 1e-5)  # noqa: E731
        d[near(y, 20)[:, :, None] | near(x, 24)[:, None, :]] = 0
    assert d.max() <= 1.6e-5 * peak
    ctx.close()
