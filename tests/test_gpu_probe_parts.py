"""Sheet velocity at points: eight warps share 32 points by panel ranges.  Point
counts at the edges of 32 and panel counts below, at and off multiples of eight,
against the oracle's panel formula.  FP64 sums of at most 2048 terms in another
order: 1e-12 of the largest velocity."""
import numpy as np
import pytest

from dvmpp_b200 import native as N
from dvmpp_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npanels", [3, 7, 8, 13, 100, 2048])
def test_points_and_panel_ranges(ctx, port, npanels):
    bx, bz = W.ellipse(npanels, 0.5, 0.3, 10.0)
    s = ctx.sim(N.Params(capacity=4096 + 8 * npanels, ux=1.5, uz=0.2), bx, bz)
    s.phase(N.PHASE_SOLVE)
    gamma = s.gamma()
    geometry = port.sheet_geometry(bx, bz)
    rng = np.random.default_rng(npanels)
    for n in (1, 31, 32, 33, 257):
        r, th = rng.uniform(0.7, 3.0, n), rng.uniform(0, 2 * np.pi, n)
        px, pz = r * np.cos(th), r * np.sin(th)
        _, _, us, ws = s.probe(px, pz)
        us0, ws0 = port.sheet_on_blobs(geometry, gamma, px, pz)
        scale = max(np.max(np.abs(us0)), np.max(np.abs(ws0)))
        assert np.max(np.abs(us - us0)) <= 1e-12 * scale
        assert np.max(np.abs(ws - ws0)) <= 1e-12 * scale
    s.close()
