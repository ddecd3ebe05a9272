"""Reconstruction at the ends of its operands' range: where WENO's weights over
a common denominator leave the exponents in which they and their reciprocal are
exact (and the quotients are formed instead), and where PPM's flattening ratio
overflows although its weight is zero."""
import numpy as np
import pytest

from oracle import Oracle
from raishinsource_b200 import config

pytestmark = pytest.mark.gpu

GRID = dict(nr=40, nth=24, nph=17)


def _region(o):
    n = o.nm1 - 1
    return (slice(n, -n),) * 3


def _stencil_max(u, axis, reach=3):
    """Largest finite magnitude among the cells of a face's stencils."""
    a = np.where(np.isfinite(u), np.abs(u), 0.0)
    m = a.copy()
    for k in range(-reach, reach + 1):
        m = np.maximum(m, np.roll(a, -k, axis))
    return m


def _compare(got, want, u, reg, tol):
    for d, axis in enumerate((2, 1, 0)):  # r, phi, theta faces of (k, j, i)
        scale = np.maximum(_stencil_max(u, axis), 1e-300)[reg]
        for side in (0, 1):
            a, b = got[2 * d + side][reg], want[2 * d + side][reg]
            assert np.array_equal(np.isnan(a), np.isnan(b))
            fin = np.isfinite(b)
            assert np.array_equal(a[~fin & ~np.isnan(b)], b[~fin & ~np.isnan(b)])
            # either way of forming the weights rounds some twenty times: 20 eps of the stencil's largest value, and
            # as much again from the smoothness indicators' own roundings
            err = np.abs(np.where(fin, a - b, 0.0)) / scale
            assert err.max() < tol, (d, side, err.max())


@pytest.mark.parametrize("irec", [config.IREC_WENO5, config.IREC_WENOZ, config.IREC_WENOM])
@pytest.mark.parametrize("lo,hi", [(-45, 5), (5, 45), (30, 75), (70, 160)])
def test_weno_states_over_the_exponent_range(gpu_ctx, irec, lo, hi):
    """Magnitudes 10^lo to 10^hi, another one in every cell, an infinity and a
    NaN among them: indicators that differ by hundreds of orders in one stencil,
    products beyond 2^500, quotients that overflow or vanish."""
    p = dict(config.torus(irec=irec, **GRID), guard=0)
    o = Oracle(p)
    o.ic_torus(seed=3)
    rng = np.random.default_rng(17)
    u = rng.standard_normal(o.prims().shape) * 10.0 ** rng.uniform(lo, hi, o.prims().shape)
    u[::7, :, ::5] = 0.0
    u[12, 8, 20, :] = np.nan
    u[15, 9, 25, :] = np.inf
    r = gpu_ctx.admit(p)
    got = r.rec2(u, cons=False)[0]
    r.release()
    _compare(got, o.rec2(u), u, _region(o), 1e-14)


def test_ppm_flattening_ratio_beyond_the_range(gpu_ctx):
    """Pressures whose fourth difference is nothing beside the second: the ratio
    overflows, and zero times it is not zero."""
    p = dict(config.torus(irec=config.IREC_PPM, **GRID), guard=0)
    o = Oracle(p)
    o.ic_torus(seed=3)
    rng = np.random.default_rng(23)
    u = 1.0 + rng.random(o.prims().shape)
    for axis, at in ((0, 12), (1, 8), (2, 20)):
        for off, value in ((-2, 1e-310), (-1, 1.0), (0, 1.5), (1, 2.0), (2, 2e-310)):
            sel = [slice(None)] * 4
            sel[axis], sel[3] = at + off, 4
            u[tuple(sel)] = value
    r = gpu_ctx.admit(p)
    got = r.rec2(u, cons=False)[0]
    r.release()
    _compare(got, o.rec2(u), u, _region(o), 1e-14)


@pytest.mark.parametrize("irec", [config.IREC_PPM, config.IREC_WENO5, config.IREC_WENOZ, config.IREC_MP5])
def test_staged_fluxes_of_rough_data_equal_direct(gpu_ctx, irec):
    """The staged kernel's own way to the face states (PPM: both cells of a face
    at once; MP5: in two passes) on data that need every limiter, against the
    direct kernel, which a source off the 16-byte boundary takes."""
    import torch
    p = dict(config.torus(irec=irec, **GRID), guard=1)
    r = gpu_ctx.admit(p)
    r.ic_torus(seed=3)
    u = r.prims()
    rng = np.random.default_rng(29)
    u *= np.where(rng.random(u.shape) < 0.3, 10.0 ** rng.uniform(-2, 2, u.shape), 1.0)
    n = u.size // 9
    src = torch.from_numpy(np.ascontiguousarray(u.reshape(n, 9).T).ravel())
    out = []
    for offset in (0, 1):
        buf = torch.zeros(9 * n + offset, dtype=torch.float64, device="cuda")
        buf[offset:] = src
        ww = torch.zeros(3, 9, *u.shape[:3], dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        r.calflx_static(buf.data_ptr() + 8 * offset, ww.data_ptr())
        m = r.nm1 - 1
        out.append(ww.cpu().numpy()[:, :, m:-m, m:-m, m:-m])
    r.release()
    a, b = out
    assert np.isfinite(a).all() and np.isfinite(b).all()
    scale = np.abs(b).max(axis=(0, 2, 3, 4))[None, :, None, None, None]
    assert (np.abs(a - b) / np.maximum(scale, 1e-300)).max() < 1e-13
