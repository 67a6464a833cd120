"""FP32 sheet velocity of a step, whose far panels stand as Gauss points in a tree, for
contours where one panel dominates a leaf of 16: 3 to 8 equal panels, remainders of
one and two panels, long straight panels among short ends, and few blobs close to
the panels, where the quadrature goes wrong first.  Against the FP64 closed form, blob
by blob.

Bound, per blob: 2e-6 of the sum over the panels of (|gamma_j| + |gamma_j+1|) times
min(1, ds / distance) / (2 pi).  A panel's closed form is rounded to FP32 in about
ten dependent operations on terms of order one (10 x 2^-24 = 6e-7, and up to three
times that where its terms cancel at some distance); the quadrature adds at most 4e-8.
Gamma comes from the free stream alone (no circulation in the wake), so both
precisions have the same.
"""
import numpy as np
import pytest

from dvmpp_b200 import native as N
from dvmpp_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _bar(nend, h=0.05):
    """A bar whose long sides are one panel each, its ends nend panels."""
    t = 2.0 * h * np.arange(1, nend + 1) / nend
    x = np.concatenate([[-0.5, 0.5], np.full(nend, 0.5), [-0.5], np.full(nend, -0.5)])
    z = np.concatenate([[-h, -h], t - h, [h], h - t])
    x[-1], z[-1] = x[0], z[0]
    return x, z


BODIES = {**{f"circle{k}": W.circle(k) for k in (3, 4, 6, 8, 17, 18, 33, 49)},
          "bar16": _bar(7), "bar42": _bar(20)}


def _points(n, bx, bz, seed):
    """Points 0.2 to 3 lengths off randomly chosen panels, outside the contour."""
    rng = np.random.default_rng(seed)
    ds = np.hypot(np.diff(bx), np.diff(bz))
    big = np.argsort(ds)[-2:]  # half of them at the longest panels and the last
    j = np.where(rng.uniform(size=n) < 0.5, rng.choice(np.append(big, ds.size - 1), n),
                 rng.integers(0, ds.size, n))
    t, off = rng.uniform(-0.5, 1.5, n), rng.uniform(0.2, 3.0, n) * ds[j]
    ex, ez = np.diff(bx)[j], np.diff(bz)[j]
    x = bx[j] + t * ex + off * ez / ds[j]  # (the contours run counter-clockwise)
    z = bz[j] + t * ez - off * ex / ds[j]
    return x, z


def _worst(ctx, bx, bz, sets):
    """Largest error of any blob of the given blob sets (one call each), in units of its
    scale (see above)."""
    got = []
    for prec in (N.F32, N.F64):
        sim = ctx.sim(N.Params(capacity=max(len(x) for x, _ in sets), precision=prec, ux=1.0, uz=0.3,
                               surface_cross=N.REFLECT), bx, bz)
        us, ws = [], []
        for x, z in sets:
            sim.set_blobs(x, z, np.zeros(len(x)), np.full(len(x), 0.01))
            sim.phase(N.PHASE_CONVECT)
            d = sim.blobs()
            us.append(d["uvs"])
            ws.append(d["wvs"])
        got.append((sim.gamma(), np.concatenate(us), np.concatenate(ws)))
        sim.close()
    gamma = got[1][0]
    assert np.array_equal(got[0][0], gamma)
    x, z = (np.concatenate(v) for v in zip(*sets))
    ds = np.hypot(np.diff(bx), np.diff(bz))
    mx, mz = 0.5 * (bx[1:] + bx[:-1]), 0.5 * (bz[1:] + bz[:-1])
    dist = np.hypot(x[:, None] - mx, z[:, None] - mz)
    scale = np.minimum(1.0, ds / dist) @ (np.abs(gamma) + np.abs(np.roll(gamma, -1))) / (2.0 * np.pi)
    err = np.hypot(got[0][1] - got[1][1], got[0][2] - got[1][2])
    return np.max(err / scale)


@pytest.mark.parametrize("n", [1, 65, 2000])
@pytest.mark.parametrize("body", BODIES)
def test_sheet_velocity_of_a_step(ctx, body, n):
    bx, bz = BODIES[body]
    assert _worst(ctx, bx, bz, [_points(n, bx, bz, n)]) <= 2e-6


@pytest.mark.parametrize("npan", [3, 4, 17, 18, 33])
def test_lone_blobs_at_the_last_panel(ctx, npan):
    """One blob per call, 0.9 to 1.3 panel lengths from the last panel's centre, to
    its outer side (the method's panels run from their collocation point on,
    src/VortexSheet.cpp:217-273, so along the contour one meets the next)."""
    bx, bz = W.circle(npan)
    ex, ez = bx[-1] - bx[-2], bz[-1] - bz[-2]
    sets = []
    for k in range(40):
        a, r = np.pi * (1 + k % 8) / 9.0, 0.9 + 0.1 * (k // 8)
        x = bx[-1] + r * (np.cos(a) * ex + np.sin(a) * ez)
        z = bz[-1] + r * (np.cos(a) * ez - np.sin(a) * ex)
        sets.append((np.array([x]), np.array([z])))
    assert _worst(ctx, bx, bz, sets) <= 2e-6
