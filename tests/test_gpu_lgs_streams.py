"""LGS frames whose uplink OTFs run on the aux stream: two LGS powfs in one
frame (64-point images, whose LLT pupils go through the FFT passes, and
32-point images, whose uplink is a launch of its own), which share that stream
and its events.

Each powfs's result depends on its own subapertures alone, so everything is
compared to the bit: the frame of both with frames of one, queued frames with
graph frames, frames in flight together with frames by themselves, and a powfs
large enough that its LLT pupils are traced beside its subapertures with one
of its first subapertures only, which traces all pupils in one launch."""
import numpy as np
import pytest

from tests.conftest import cuda_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")]

ISIMS = (3, 41, 200)


def _add(ctx, nsa, N, nwfs):
    from maos_b200 import shwfs
    nopd, pix = N // 2, 6
    rng = np.random.default_rng(N)
    side, dsa, hs = 52, 0.5, 90e3
    ip = ctx.powfs_add(nsa=nsa, nopd=nopd, embfac=2, notf=N, pixpsax=pix, pixpsay=pix, pixthetax=1e-6, pixthetay=1e-6,
                       wvl=0.6e-6, dsa=dsa, dx=dsa / nopd, areascale=1.0, hs=hs, has_etf=1, has_llt=1, llt_nx=nopd,
                       llt_ox=7.0, gradtype=shwfs.SHWFS_GRAD_COG, sigmatch=1)
    i = np.arange(nsa)
    ctx.powfs_set_geom(ip, (i % side - side / 2) * dsa, (i // side - side / 2) * dsa, np.ones(nsa * nopd * nopd), np.ones(nsa))
    f = np.fft.fftfreq(N)
    etf = np.exp(-30 * f[:, None] ** 2 - 60 * f[None] ** 2).astype(complex)
    ctx.powfs_set_etf(ip, np.broadcast_to(etf.ravel(), (nsa, N * N)))
    ctx.powfs_set_lltamp(ip, np.ones((nopd, nopd)) / nopd)
    p = (np.arange(pix) - pix // 2) * 2 % N
    idx = np.full((pix * pix, 4), -1)
    idx[:, 0] = (p[:, None] * N + p[None]).ravel()
    ctx.powfs_set_simap(ip, idx, np.ones((pix * pix, 4)))
    for k in range(nwfs):
        t = 35 / 206265 * np.exp(2j * np.pi * (k + 0.3) / nwfs)
        ctx.wfs_add(ipowfs=ip, thetax=t.real, thetay=t.imag, hs=hs, hc=0.0, misregx=0.0, misregy=0.0, sigsim=700.0,
                    wvlwt=1.0, noisy=int(rng.integers(0, 2)))


def _context(*powfs):
    from maos_b200 import shwfs
    rng = np.random.default_rng(5)
    ctx = shwfs.Context(0)
    ctx.set_dt(1 / 800)
    n, dx = 512, 1 / 16
    scr = []
    for _ in range(3):
        s = np.cumsum(np.cumsum(rng.standard_normal((n, n)), 0), 1)
        scr.append(1e-6 * s / np.abs(s).max())
    ctx.atm_set([dict(nx=n, ny=n, dx=dx, ox=-n / 2 * dx, oy=-n / 2 * dx, ht=4e3 * k, vx=9.0 - k, vy=4.0 + k, alpha=1.0)
                 for k in range(3)], scr)
    for nsa, N, nwfs in powfs:
        _add(ctx, nsa, N, nwfs)
    return ctx


def _frames(ctx, i0, i1, ngrad, how="frame_queue"):
    out = []
    for isim in ISIMS:
        getattr(ctx, how)(isim, i0, i1)
        g = np.zeros(ngrad)
        ctx.frame_sync_range(i0, i1, out=g)
        out.append(g)
    return np.stack(out)


@pytest.mark.parametrize("nsa", [60, 2400])  # of 32x32 points, 3 layers: below and above 16384 gathers per SM
def test_two_lgs_powfs_in_one_frame(nsa):
    na, nb = 2 * (2 * nsa), 3 * (2 * 150)
    ctx = _context((nsa, 64, 2), (150, 32, 3))
    both = _frames(ctx, 0, 5, na + nb)
    assert np.isfinite(both).all() and (both != 0).mean() > 0.9
    assert np.array_equal(both[:, :na], _frames(ctx, 0, 2, na))
    assert np.array_equal(both[:, na:], _frames(ctx, 2, 5, nb))
    ctx.frame_graph(ISIMS[0], 0, 5)  # the warm-up frame
    assert np.array_equal(both, _frames(ctx, 0, 5, na + nb, "frame_graph"))
    for isim in (7, 8, 9, ISIMS[-1]):  # nothing waits on the host between these
        ctx.frame_queue(isim, 0, 5)
    g = np.zeros(na + nb)
    ctx.frame_sync_range(0, 5, out=g)
    assert np.array_equal(both[-1], g)
    ctx.close()


def test_llt_beside_the_trace_equals_one_launch():
    big, few = _context((2400, 64, 2)), _context((60, 64, 2))
    a, b = _frames(big, 0, 2, 2 * 2 * 2400), _frames(few, 0, 2, 2 * 2 * 60)
    big.close()
    few.close()
    a = a.reshape(len(ISIMS), 2, 2, 2400)[..., :60]  # frame, sensor, axis, subaperture
    assert np.array_equal(a, b.reshape(len(ISIMS), 2, 2, 60))


def test_llt_chain_is_booked_as_uplink():
    """The ray-trace stage times the subapertures' trace alone, also where the LLT pupils are traced beside it."""
    ctx = _context((2400, 64, 2))
    _frames(ctx, 0, 2, 2 * 2 * 2400)
    ctx.profile_enable(True)
    ctx.profile_read()
    ctx.frame_queue(3, 0, 2)
    stages = ctx.profile_read()
    ctx.close()
    assert stages["raytrace"][1] == 1 and stages["uplink"][1] == 2
