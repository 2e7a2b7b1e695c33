"""Science wavefront sums against a plain FP64 evaluation, from an aperture
inside one 16x16 tile to launches of more blocks than the chip holds at once
(one, two and four batches of tiles per block of evl_sums_kernel).

Tolerance: with unit total amplitude each of sum a o^2, (sum a o)^2 and the
tip/tilt part changes by at most 2 eps peak^2 where the traced OPD is off by
eps peak (eps = 1.6e-5, the bound of the trace tests for one layer), and an
error is a difference of two of them: 4 eps peak^2."""
import numpy as np
import pytest

from tests.conftest import cuda_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")]


@pytest.mark.parametrize("side,nevl", [(5, 1), (17, 2), (143, 1), (143, 110), (143, 1000), (300, 9)])
def test_wavefront_sums(side, nevl):
    from maos_b200 import shwfs
    rng = np.random.default_rng(side + nevl)
    n, sdx, dx, ht = 64, 0.25, 1 / 16, 1000.0
    scr = 1e-6 * rng.standard_normal((n, n))
    X, Y = np.meshgrid(np.arange(side), np.arange(side))
    keep = (X - side / 2) ** 2 + (Y - side / 2) ** 2 <= (side / 2) ** 2
    x, y = (X[keep] - side / 2) * dx, (Y[keep] - side / 2) * dx
    amp = rng.uniform(0, 1, len(x))
    amp /= amp.sum()
    theta = [(1e-4 * k, -2e-4 * k) for k in range(nevl)]
    ctx = shwfs.Context(0)
    ctx.set_dt(1 / 800)
    ctx.atm_set([dict(nx=n, ny=n, dx=sdx, ox=-n / 2 * sdx, oy=-n / 2 * sdx, ht=ht, vx=0.0, vy=0.0, alpha=1.0)], [scr])
    ctx.evl_set_aper(x, y, dx, amp)
    for t in theta:
        ctx.evl_add_dir(*t)
    ctx.evl_queue(0, do_psf=False)
    wfe, coeff = ctx.evl_sync()
    ctx.close()
    B = np.stack([np.ones_like(x), x, y])
    A = np.linalg.inv((B * amp) @ B.T)
    tol = 4 * 1.6e-5 * np.abs(scr).max() ** 2
    for k in sorted({0, nevl // 2, nevl - 1}):
        u, v = (x + ht * theta[k][0]) / sdx + n / 2, (y + ht * theta[k][1]) / sdx + n / 2
        ju, jv = np.floor(u).astype(int), np.floor(v).astype(int)
        at = lambda a, b: scr[a % n, b % n]  # noqa: E731
        o = (at(jv, ju) * (1 - u + ju) + at(jv, ju + 1) * (u - ju)) * (1 - v + jv) + (
            at(jv + 1, ju) * (1 - u + ju) + at(jv + 1, ju + 1) * (u - ju)) * (v - jv)
        b = (B * amp) @ o
        tot, pis, ptt = (amp * o * o).sum(), b[0] ** 2, b @ A @ b
        assert np.abs(wfe[k] - [tot - pis, ptt - pis, tot - ptt]).max() <= tol
        # one mode's coefficient is the sums times a row of the inverse moments
        assert np.abs(coeff[k] - A @ b).max() <= 1.6e-5 * np.abs(scr).max() * np.abs(A @ (B * amp)).sum(1).max()
