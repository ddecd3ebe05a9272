"""The FP32 faces of a mixed run keep their arithmetic: every constant evaluated
in FP32, IEEE quotients in WENO and PPM, the same roundings whichever kernel
forms a face.  MP5 chooses between the unlimited and the limited value by an
absolute 1e-10, far below FP32's resolution, so that a last bit in every face
becomes a jump of percents of the small theta velocity in a few of many cells."""
import numpy as np
import pytest

from raishinsource_b200 import Context, config

pytestmark = pytest.mark.gpu

SCHEMES = [config.IREC_PPM, config.IREC_MP5, config.IREC_WENO5, config.IREC_WENOZ]

# Signed sums over the stored cells, in units of each field's maximum, of rho,
# u1, u2, u3, p, b1, b2, b3 after one mixed step, as the direct kernel
# gave them when it formed each quotient and constant in FP32 at each face.
SUMS = {
    ('3d', 5):
    (-0.220817762788, -0.384122977629, -0.584466529339, -6.47486229816, -0.406982781067, -0.659157451588, 1.82717040312, -1.40164993367),
    ('3d', 6):
    (-0.730052412321, -0.070584517006, 0.861820572067, -9.64966945287, -0.646857216769, -0.0395598783387, 3.1453292827, -0.944594021793),
    ('3d', 7):
    (-0.727448702007, -3.09935317012, -3.30789906079, 5.45704163428, -0.649646450269, -0.040918497067, 5.28256461436, -0.951124456953),
    ('3d', 9):
    (-0.72659704128, -3.12295022428, -3.53652200364, -1.07213029622, -0.650150212937, -0.038774146718, 4.95643791723, -0.953530864875),
    ('2d', 5):
    (-1.17093347054, -1.23315187929, -1.65040449548, -0.0096860826661, -1.13807583127, -2.14223186822, -0.906778554701, 0.492054757601),
    ('2d', 6):
    (-1.17134870613, -0.689921125521, -1.10110912182, 1.20881914584, -1.1469180972, -2.14370741552, 1.52220853222, 0.492497240641),
    ('2d', 7):
    (-1.17138665954, -0.567328124943, -0.910764578606, -1.71858960345, -1.14612838516, -2.14488481674, 0.363787856605, 0.491444614439),
    ('2d', 9):
    (-1.17135219519, -0.998409246194, -1.46733765382, 1.247722286, -1.1461573092, -2.14512010478, 0.400329347276, 0.491505008093),
}
GRIDS = {"3d": dict(nr=40, nth=24, nph=16), "2d": dict(nr=64, nth=64)}
# FP64 roundings move a sum by 1e-14 of the maximum a cell at most, 1e-12 or so
# over 15,360 cells; a last bit of the FP32 faces moved u1's by 4e-8 at least.
TOL_SUM = 1e-9


@pytest.mark.parametrize("irec", SCHEMES)
@pytest.mark.parametrize("grid", ["3d", "2d"])
def test_one_mixed_step_as_recorded(gpu_ctx, grid, irec):
    r = gpu_ctx.admit(dict(config.torus(irec=irec, precision="mixed", **GRIDS[grid]), guard=1))
    r.ic_torus_device(seed=11, beta=100.0, rmax=12.0)
    r.step(1, strict=False)
    x = r.stored_prims().reshape(9, -1)[[0, 1, 2, 3, 4, 6, 7, 8]]
    r.release()
    sign = np.where((np.arange(x.shape[1]) * 2654435761 % 2**32) >> 31, 1.0, -1.0)
    got = (sign * x).sum(axis=1) / np.maximum(np.abs(x).max(axis=1), 1e-300)
    assert np.abs(got - SUMS[grid, irec]).max() < TOL_SUM, got - SUMS[grid, irec]


@pytest.fixture(scope="module")
def direct_ctx():
    """A context whose runs read the stencil from global memory."""
    mp = pytest.MonkeyPatch()
    mp.setenv("RAISHIN_FLUX_TMA", "0")
    ctx = Context(0)
    mp.undo()
    yield ctx
    ctx.close()


# One interior cell a direction, ragged rows of a tile, several tiles along r.
@pytest.mark.parametrize("irec", SCHEMES)
@pytest.mark.parametrize("nr,nth,nph", [(12, 12, 16), (40, 13, 17), (68, 23, 19)])
def test_staged_fp32_faces_equal_direct(gpu_ctx, direct_ctx, irec, nr, nth, nph):
    """The FP32 faces are the same bits in both kernels; the FP64 faces inside
    2 r_H may differ in a last bit, 1e-14 of a field, so one differing FP32
    rounding (6e-8 of a face's flux) stands out."""
    p = dict(config.torus(nr=nr, nth=nth, nph=nph, irec=irec, precision="mixed"), guard=1)
    out = []
    for ctx in (gpu_ctx, direct_ctx):
        r = ctx.admit(p)
        r.ic_torus(seed=7)
        r.step(1, strict=False)
        out.append(r.stored_prims().reshape(9, -1))
        r.release()
    a, b = out
    assert np.isfinite(a).all()
    scale = np.maximum(np.abs(b).max(axis=1), 1e-300)
    scale[1:4] = scale[1:4].max()  # the theta velocity is a thousandth of the others
    assert (np.abs(a - b).max(axis=1) / scale).max() < 1e-12
