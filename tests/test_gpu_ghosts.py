"""The one-pass ghost fill (every code that copies, mirrors, zeroes or wraps an
interior cell) against the oracle's passes, value for value, at the smallest
extents it takes and just below them, where the separate passes run."""
import numpy as np
import pytest

from oracle import Oracle
from raishinsource_b200 import config

pytestmark = pytest.mark.gpu

NM1 = 4  # MP5 with flux-CT


def _codes(inner_r, outer_r, inner_t, outer_t):
    """Codes that differ between variables, so that each takes its own source."""
    rows = [[inner_r[v % len(inner_r)] for v in range(9)], [outer_r[v % len(outer_r)] for v in range(9)], [1] * 9, [1] * 9,
            [inner_t[v % len(inner_t)] for v in range(9)], [outer_t[v % len(outer_t)] for v in range(9)]]
    return rows


@pytest.mark.parametrize("codes", [
    config.torus_bcs(),
    _codes([5, 14, 12], [5, 18, 13], [14, 12, 5], [12, 14, 13]),
    _codes([13], [14, 12], [5], [5, 13]),
])
# interior cells along (r, phi, theta): nm1 (the least of one pass), one less, ragged
@pytest.mark.parametrize("cells", [(4, 4, 4), (3, 4, 4), (4, 3, 4), (4, 4, 3), (33, 5, 9), (8, 1, 7)])
def test_one_pass_equals_the_passes(gpu_ctx, codes, cells):
    nr, nph, nth = (n + 2 * NM1 for n in cells)
    p = dict(config.torus(nr=nr, nth=nth, nph=nph), guard=1, ibc=codes, flags=config.FLAG_FULL)
    o = Oracle(p)
    o.ic_torus(seed=5)
    rng = np.random.default_rng(nr + 7 * nph + 31 * nth)
    u = rng.standard_normal(o.prims().shape)
    r = gpu_ctx.admit(p)
    got, want = r.bnd_part("bnd4", u, u), o.bnd_part("bnd4", u, u)
    r.release()
    assert np.array_equal(got, want)
