"""FP32 sheet velocity and right-hand side over the trees (of the blobs and of the
panels) against the FP64 path, at the sizes where they can go wrong: panel
counts around a panel leaf (16), a right-hand-side group (32) and a block's
share of the tree (256 panels), few and no blobs, blobs at the surface and far
away.  Bounds: the FP32 path's 1e-5 relative L2 for fields and gamma."""
import numpy as np
import pytest

from dvmpp_b200 import native as N
from dvmpp_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _blobs(n, seed, sigma):
    x, z, g, s = W.wake(n, seed, sigma)
    k = n // 10  # some close to the surface, some far away
    rng = np.random.default_rng(seed)
    t = rng.uniform(0, 2 * np.pi, k)
    r = 0.5 + 10.0 ** rng.uniform(-4, -1, k)
    x[:k], z[:k] = r * np.cos(t), r * np.sin(t)
    x[k:2 * k] += 500.0
    return x, z, g, s


@pytest.mark.parametrize("npan,n", [(3, 100), (15, 100), (16, 1000), (17, 65), (31, 3000), (33, 3000),
                                    (255, 5000), (257, 5000), (1024, 20000), (2047, 2000), (64, 0),
                                    (64, 1), (128, 40000)])
def test_sheet_and_rhs_match_fp64(ctx, npan, n):
    bx, bz = W.circle(npan)
    blobs = _blobs(n, npan + n, 0.03) if n else [np.zeros(0)] * 4
    got = []
    for prec in (N.F32, N.F64):
        sim = ctx.sim(N.Params(capacity=max(n, 1), precision=prec, ux=1.0, uz=0.3), bx, bz)
        sim.set_blobs(*blobs)
        sim.phase(N.PHASE_SOLVE)
        sim.phase(N.PHASE_SHEETBC)
        d = sim.blobs()
        got.append((sim.gamma(), sim.rhs(), d["uvs"], d["wvs"]))
        sim.close()
    for a, b in zip(got[0], got[1]):
        assert np.all(np.isfinite(a))
        assert np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(b) + 1e-300
