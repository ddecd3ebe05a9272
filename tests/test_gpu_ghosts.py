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


@pytest.mark.parametrize("codes", [
    _codes([13, 5], [13, 18], [12], [12]),   # a zero of the r pass is negated by the theta pass
    _codes([12], [14, 18], [13, 12], [12, 5]),
])
def test_one_pass_keeps_the_sign_of_zero(gpu_ctx, codes):
    p = dict(config.torus(nr=20, nth=19, nph=13), guard=1, ibc=codes, flags=config.FLAG_FULL)
    o = Oracle(p)
    o.ic_torus(seed=5)
    u = np.random.default_rng(11).standard_normal(o.prims().shape)
    u[::3] = 0.0
    r = gpu_ctx.admit(p)
    got, want = r.bnd_part("bnd4", u, u), o.bnd_part("bnd4", u, u)
    r.release()
    assert (np.signbit(want) & (want == 0)).any()
    assert np.array_equal(got, want) and np.array_equal(np.signbit(got), np.signbit(want))


def test_batched_passes_equal_the_oracle(gpu_ctx):
    """A batch with a member whose codes need the separate passes (fixed, linear,
    parabolic and difference-keeping radial ghosts, other codes for other
    variables): its ghost tiles take one variable each, and the members whose
    codes one pass could fill take them too.  Against the oracle, step by step,
    and bit for bit against the same runs alone."""
    odd = [[5, 4, 3, 5, 5, 2, 7, 2, 4], [2, 18, 18, 4, 3, 5, 7, 5, 2], [1] * 9, [1] * 9,
           [14, 14, 14, 12, 14, 5, 14, 13, 12], [14, 14, 14, 12, 14, 5, 2, 14, 12]]
    params = [dict(config.torus(nr=48, nth=40), guard=1, ibc=odd), dict(config.torus(nr=36, nth=44), guard=1)]
    oracles = [Oracle(p) for p in params]
    batch, alone = [gpu_ctx.admit(p) for p in params], [gpu_ctx.admit(p) for p in params]
    for n, o in enumerate(oracles):
        o.ic_torus(seed=40 + n)
        o.init_cons()
        for r in (batch[n], alone[n]):
            r.upload_prims(o.prims())
    for _ in range(3):
        for o in oracles:
            o.step(1)
        gpu_ctx.step_batch(batch, 1)
        for a, b, o in zip(alone, batch, oracles):
            a.step(1)
            got, want = b.prims(), o.prims()
            assert np.array_equal(a.prims(), got)
            scale = np.maximum(np.abs(want).reshape(-1, 9).max(axis=0), 1e-300)
            assert (np.abs(got - want).reshape(-1, 9).max(axis=0) / scale).max() < 1e-12  # the per-step parity bound
            a.upload_prims(want, t0=o.time)
            b.upload_prims(want, t0=o.time)
    for r in batch + alone:
        r.release()
