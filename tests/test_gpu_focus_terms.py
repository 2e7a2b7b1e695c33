"""Focus terms of the WFS OPD (shwfs_wfs_set_opd_terms) against their
definition, f ((x - a)^2 + (y - b)^2) less its mean over the pupil points, for
pupils of both trace kernels and after a change of geometry.

Tolerance: the polynomial is evaluated in FP64 from sums of the pupil points,
rounded to FP32 and added to a zero OPD: half a unit in the last place of the
largest value, 2^-24 of it, and as much again for the FP64 part."""
import numpy as np
import pytest

from tests.conftest import cuda_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")]


@pytest.mark.parametrize("nopd", [16, 20, 32])
def test_focus_terms(nopd):
    import torch
    from maos_b200 import shwfs
    rng = np.random.default_rng(nopd)
    nsa, dx, a, b = 37, 0.03, 8.0, -1.5
    ctx = shwfs.Context(0)
    ip = ctx.powfs_add(nsa=nsa, nopd=nopd, embfac=1, notf=0, pixpsax=0, pixpsay=0, dsa=nopd * dx, dx=dx, hs=np.inf,
                       areascale=1.0, wvl=1e-6, llt_ox=a, llt_oy=b, gradtype=shwfs.SHWFS_GRAD_ZTILT)
    iw = ctx.wfs_add(ipowfs=ip, thetax=0.0, thetay=0.0, hs=np.inf, hc=0.0, misregx=0.0, misregy=0.0, sigsim=1.0,
                     wvlwt=1.0, noisy=0)
    ctx.atm_set([dict(nx=32, ny=32, dx=1.0, ox=-16.0, oy=-16.0, ht=0.0, vx=0.0, vy=0.0, alpha=1.0)], [np.zeros((32, 32))])
    opd = torch.zeros(nsa * nopd * nopd, device="cuda")
    torch.cuda.synchronize()
    for _ in range(2):  # the second geometry replaces the first
        ox, oy = rng.uniform(-15, 15, nsa), rng.uniform(-12, 15, nsa)
        ctx.powfs_set_geom(ip, ox, oy, np.ones(nsa * nopd * nopd))
        x = (ox[:, None, None] + np.arange(nopd) * dx) + np.zeros((1, nopd, 1))
        y = (oy[:, None, None] + np.arange(nopd)[:, None] * dx) + np.zeros((1, 1, nopd))
        for tel, llt in ((3e-9, 0.0), (0.0, -2e-9), (3e-9, -2e-9)):
            ctx.wfs_set_opd_terms(iw, focus_tel=tel, focus_llt=llt)
            ctx.raytrace_dev(iw, 0, opd)
            ctx.sync()
            r, q = x * x + y * y, (x - a) ** 2 + (y - b) ** 2
            ref = tel * (r - r.mean()) + llt * (q - q.mean())
            got = opd.double().cpu().numpy().reshape(ref.shape)
            assert np.abs(got - ref).max() <= 2 ** -23 * np.abs(ref).max()
    ctx.close()
