"""The staged face kernel (one thread per face, stencil in shared memory) and
the branch-free divisions of the face states, at the sizes and operands where
they can go wrong."""
import numpy as np
import pytest

from oracle import Oracle
from raishinsource_b200 import Context, config

pytestmark = pytest.mark.gpu

TOL = 1e-12  # of each field's maximum, as every per-step parity test


@pytest.fixture(scope="module")
def direct_ctx():
    """A context whose runs read the stencil from global memory."""
    mp = pytest.MonkeyPatch()
    mp.setenv("RAISHIN_FLUX_TMA", "0")
    ctx = Context(0)
    mp.undo()
    yield ctx
    ctx.close()


# A tile is 32 faces along i and four rows along phi (theta faces: along
# theta): one interior cell, rows that end inside a tile, a second tile of one
# column along i (nm0 = 3: 33 faces from 40 - 2) and a run of several tiles.
@pytest.mark.parametrize("irec", [config.IREC_PPM, config.IREC_MP5, config.IREC_WENO5, config.IREC_WENOZ,
                                  config.IREC_WENOM])
@pytest.mark.parametrize("nr,nth,nph", [(12, 12, 16), (40, 13, 17), (36, 14, 18), (68, 23, 19)])
def test_staged_faces_equal_direct(gpu_ctx, direct_ctx, irec, nr, nth, nph):
    p = dict(config.torus(nr=nr, nth=nth, nph=nph, irec=irec), guard=1)
    out = []
    for ctx in (gpu_ctx, direct_ctx):
        r = ctx.admit(p)
        r.ic_torus(seed=7)
        r.step(2, strict=False)
        out.append(r.stored_prims())
        r.release()
    a, b = out
    assert np.isfinite(a).all()
    err = np.abs(a - b).reshape(9, -1).max(axis=1) / np.maximum(np.abs(b).reshape(9, -1).max(axis=1), 1e-300)
    # two steps; the theta velocity is a thousandth of the others, so its error is taken against the largest velocity
    vmax = np.abs(b[1:4]).max()
    err[1:4] = np.abs(a[1:4] - b[1:4]).reshape(3, -1).max(axis=1) / vmax
    assert err.max() < TOL, err


@pytest.mark.parametrize("value", [0.0, 1e-300, 1e-160, 1e140])
def test_face_states_outside_the_fast_range(gpu_ctx, value):
    """Pressures whose quotients leave the branch-free operators' exponent
    range (2^-500 to 2^500, or zero): the face states take the IEEE operators
    and equal the oracle's."""
    p = dict(config.torus(nr=24, nth=20, nph=12, irec=config.IREC_MINMOD), guard=0)
    o = Oracle(p)
    o.ic_torus(seed=3)
    u = o.prims()
    u[:, :, ::3, 4] = value
    r = gpu_ctx.admit(p)
    got, want = r.calflx(u), o.fluxes(u)
    r.release()
    n = o.nm1 - 1
    a, b = got[n:-n, n:-n, n:-n], want[n:-n, n:-n, n:-n]
    assert np.array_equal(np.isfinite(a), np.isfinite(b))
    scale = np.abs(b).reshape(-1, 9, 3).max(axis=(0, 2))
    err = np.abs(a - b).reshape(-1, 9, 3).max(axis=(0, 2)) / np.maximum(scale, 1e-300)
    assert err.max() < TOL, err
