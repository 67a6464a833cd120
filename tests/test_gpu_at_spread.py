"""FP32 velocities at targets that do not lie together, and at sets with non-finite
targets.  A block holds its 256 targets' offsets from one of them, so a far neighbour
must not cost a target precision, nor a NaN its result.

Bounds: a lone source's term is rounded in its two offsets (2^-24 each), r^2, the
reciprocal (2^-22), the core kernel and the products: below 16 x 2^-24 = 1e-6
relative for the sources 1e-4 from their targets, whose pair dominates everything else
by the ratio of the distances.  A target among non-finite ones gives what it gives
among finite ones to the FP32 bar of 1e-5."""
import numpy as np
import pytest

from dvmpp_b200 import native as N
from dvmpp_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nt", [2, 33, 256, 300])
@pytest.mark.parametrize("spread,r", [(1.0, 1e-4), (10.0, 1e-4), (100.0, 1e-4), (1e3, 1e-3),
                                      (1e3, 1e-4), (1e5, 1e-4), (1e12, 1e6)])
def test_far_neighbours_cost_nothing(ctx, spread, r, nt):
    rng = np.random.default_rng(nt)
    tx, tz = rng.uniform(0.0, spread, (2, nt))
    a = rng.uniform(0.0, 2.0 * np.pi, nt)
    sx, sz = tx + r * np.cos(a), tz + r * np.sin(a)
    g, s = 1e-3 * rng.choice([-1.0, 1.0], nt) * rng.uniform(0.5, 1.0, nt), np.full(nt, 0.1 * r)
    s[::2] = 3.0 * r  # half of the pairs inside a core
    u, w = ctx.biot_savart_at(sx, sz, g, s, tx, tz, N.F32)
    u0, w0 = ctx.biot_savart_at(sx, sz, g, s, tx, tz, N.F64)
    assert np.max(np.hypot(u - u0, w - w0) / np.hypot(u0, w0)) <= 1e-6


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("where", [[0], [0, 1, 2, 256], [255, 256], [40]])
def test_non_finite_targets_spoil_only_themselves(ctx, where, bad):
    x, z, g, s = W.wake(700, 3, 0.06)
    tx, tz = W.collocation_circle(300)
    u0, w0 = ctx.biot_savart_at(x, z, g, s, tx, tz, N.F64)
    bx, bz = tx.copy(), tz.copy()
    bx[where] = bad
    bz[where[-1]] = bad
    u, w = ctx.biot_savart_at(x, z, g, s, bx, bz, N.F32)
    ok = np.setdiff1d(np.arange(300), where)
    assert np.linalg.norm(u[ok] - u0[ok]) <= 1e-5 * np.linalg.norm(u0[ok])
    assert np.linalg.norm(w[ok] - w0[ok]) <= 1e-5 * np.linalg.norm(w0[ok])


@pytest.mark.parametrize("npan,n", [(3, 100), (15, 1000), (16, 1), (17, 65), (31, 3000), (33, 3000),
                                    (128, 5000), (129, 5000), (255, 5000), (257, 20000), (2047, 2000),
                                    (64, 0)])
def test_right_hand_side_over_the_tree(ctx, npan, n):
    """The right-hand side of a stage (always over the blobs' tree), blobs down to 1e-7
    panel lengths from collocation points among them: entry by entry, relative to
    the sum of the absolute terms (16 x 2^-24 and the expansions' 2^-24)."""
    bx, bz = W.circle(npan)
    xc, zc = 0.5 * (bx[1:] + bx[:-1]), 0.5 * (bz[1:] + bz[:-1])
    rng = np.random.default_rng(npan + n)
    x, z, g, s = W.wake(n, npan + n, 0.03) if n else [np.zeros(0)] * 4
    k = n // 4
    j = rng.integers(0, npan, k)
    r, a = 10.0 ** rng.uniform(-8.0, -1.0, k), rng.uniform(0.0, 2.0 * np.pi, k)
    x[:k], z[:k], s[:k] = xc[j] + r * np.cos(a), zc[j] + r * np.sin(a), 0.1 * r
    got = []
    for prec in (N.F32, N.F64):
        sim = ctx.sim(N.Params(capacity=max(n, 1), precision=prec, ux=1.0, uz=0.3), bx, bz)
        sim.set_blobs(x, z, g, s)
        sim.phase(N.PHASE_CONVECT)
        got.append(sim.rhs())
        sim.close()
    d2 = np.full(npan, 0.0)
    for c0 in range(0, n, 1000):
        q = np.hypot(xc[:, None] - x[c0:c0 + 1000], zc[:, None] - z[c0:c0 + 1000])
        d2 += np.sum(np.abs(g[c0:c0 + 1000]) / q, axis=1)
    scale = np.append(1.1 + d2 / (2.0 * np.pi), np.sum(np.abs(g)) + 1e-300)
    assert np.max(np.abs(got[0] - got[1]) / scale) <= 1.1e-6
