"""FP32 solve and sheet velocity called alone: pair by pair up to a size, over a tree
above it, and in a step always over the tree.  Both sides of each line, bodies whose
right-hand side takes groups of eight points and of 32, against an FP64 simulation
of the same state.

Tolerances: the right-hand side and the panel terms are rounded to FP32 once each
(2^-24 relative to their largest terms, accumulated in FP64 or compensated) and the
right-hand side is a small rest of them: 1e-5 of the largest gamma and velocity, the
bound of the other FP32 sheet tests.
"""
import numpy as np
import pytest

from dvmpp_b200 import native as N
from dvmpp_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npanels,n,capacity", [
    (7, 1000, 4096), (64, 63, 4096), (128, 4097, 8192), (129, 4097, 8192),
    (256, 5000, 1 << 18), (256, 5000, 1 << 19), (257, 5000, 8192), (1024, 5000, 1 << 18),
    (1024, 5000, 1 << 19)])
def test_alone_matches_fp64(ctx, npanels, n, capacity):
    bx, bz = W.ellipse(npanels, 0.5, 0.3, 10.0)
    x, z, g, sg = W.wake(n, 3, W.core_size(bx, bz))
    out = []
    for prec in (N.F32, N.F64):
        s = ctx.sim(N.Params(capacity=capacity, precision=prec, ux=1.0, uz=0.2), bx, bz)
        s.set_blobs(x, z, g, sg)
        s.phase(N.PHASE_SOLVE)
        s.phase(N.PHASE_SHEETBC)
        d = s.blobs()
        out.append((s.gamma(), d["uvs"], d["wvs"]))
        s.close()
    for a, b in zip(*out):
        assert np.max(np.abs(a - b)) <= 1e-5 * max(np.max(np.abs(b)), 1e-3)


@pytest.mark.parametrize("npanels", [8, 63, 128, 129, 300])
def test_step_right_hand_side(ctx, npanels):
    """Gamma of a whole step, whose right-hand side comes from the tree."""
    bx, bz = W.ellipse(npanels, 0.5, 0.3, 10.0)
    x, z, g, sg = W.wake(6000, 4, W.core_size(bx, bz))
    out = []
    for prec in (N.F32, N.F64):
        s = ctx.sim(N.Params(capacity=8192 + 8 * npanels, precision=prec, rng=N.RNG_PHILOX,
                             ux=1.0, seed=5), bx, bz)
        s.set_blobs(x, z, g, sg)
        s.step(1)
        out.append(s.gamma())
        s.close()
    assert np.max(np.abs(out[0] - out[1])) <= 1e-5 * np.max(np.abs(out[1]))
