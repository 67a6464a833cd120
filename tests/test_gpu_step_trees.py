"""What a step sums over the trees of blobs and panels in FP32 -- a call of the solve or of
the sheet velocity alone goes by pairs up to some size -- against FP64, at panel
counts around a panel leaf (16), a right-hand-side group (8 or 32) and a block's share of
the tree (256), with no, one and many blobs, blobs at the surface and far away.

Bounds: gamma, right-hand side and sheet velocity 1e-5 relative L2, the FP32 path's bar.
The sheet velocity of each blob, against the FP64 sum with the same gamma: 2e-6 of the sum
over the panels of (|gamma_j| + |gamma_j+1|) min(1, ds / distance) (1 + log(ds / distance
to a panel's end), where that is positive) / (2 pi), as for a panel's closed form in FP32
and the quadrature, and 4 x 2^-24 sqrt(np) max |gamma| for the order-one terms that
cancel in far panels' closed forms (a leaf spread wider than its panels sums them all)."""
import numpy as np
import pytest

from dvmpp_b200 import native as N
from dvmpp_b200 import workloads as W

pytestmark = pytest.mark.gpu

CASES = [(3, 100), (15, 100), (16, 1000), (17, 65), (31, 3000), (32, 3000), (33, 3000), (128, 1), (129, 1),
         (255, 5000), (256, 5000), (257, 5000), (1024, 20000), (2047, 2000), (64, 0), (64, 1), (128, 40000)]


def _blobs(n, seed, far):
    if n == 0:
        return [np.zeros(0)] * 4
    x, z, g, s = W.wake(n, seed, 0.03)
    k = n // 10
    rng = np.random.default_rng(seed)
    t = rng.uniform(0, 2 * np.pi, k)
    r = 0.5 + 10.0 ** rng.uniform(-4, -1, k)
    x[:k], z[:k] = r * np.cos(t), r * np.sin(t)
    if far:
        x[k:2 * k] += 500.0
    return x, z, g, s


def _stage(ctx, prec, bx, bz, blobs, gamma=None):
    sim = ctx.sim(N.Params(capacity=max(len(blobs[0]), 1), precision=prec, ux=1.0, uz=0.3), bx, bz)
    sim.set_blobs(*blobs)
    if gamma is None:
        sim.phase(N.PHASE_CONVECT)
    else:
        sim.set_gamma(gamma)
        sim.phase(N.PHASE_SHEETBC)
    d = sim.blobs()
    out = sim.gamma(), sim.rhs(), d["uvs"], d["wvs"]
    sim.close()
    return out


@pytest.mark.parametrize("npan,n", CASES)
def test_stage_matches_fp64(ctx, npan, n):
    bx, bz = W.circle(npan)
    blobs = _blobs(n, npan + n, True)
    for a, b in zip(_stage(ctx, N.F32, bx, bz, blobs), _stage(ctx, N.F64, bx, bz, blobs)):
        assert np.all(np.isfinite(a))
        assert np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(b) + 1e-300


@pytest.mark.parametrize("npan,n", [c for c in CASES if c[1] > 0])
def test_sheet_velocity_of_each_blob(ctx, npan, n):
    bx, bz = W.circle(npan)
    blobs = _blobs(n, npan + n, False)
    gamma, _, u, w = _stage(ctx, N.F32, bx, bz, blobs)
    _, _, u0, w0 = _stage(ctx, N.F64, bx, bz, blobs, gamma)
    ds = np.hypot(np.diff(bx), np.diff(bz))
    mx, mz = 0.5 * (bx[1:] + bx[:-1]), 0.5 * (bz[1:] + bz[:-1])
    weight = np.abs(gamma) + np.abs(np.roll(gamma, -1))
    bound = np.empty(n)
    for c in range(0, n, 2000):
        x, z = blobs[0][c:c + 2000, None], blobs[1][c:c + 2000, None]
        # (a panel runs from its collocation point on, src/VortexSheet.cpp:217-273)
        end = np.minimum(np.hypot(x - mx, z - mz), np.hypot(x - mx - np.diff(bx), z - mz - np.diff(bz)))
        log = 1.0 + np.maximum(0.0, np.log(ds / end))
        bound[c:c + 2000] = 2e-6 / (2.0 * np.pi) * (np.minimum(1.0, ds / end) * log) @ weight
    bound += 4.0 * 2.0 ** -24 * np.sqrt(npan) * np.max(np.abs(gamma))
    err = np.hypot(u - u0, w - w0)
    assert np.max(err / bound) <= 1.0
