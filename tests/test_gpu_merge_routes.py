"""Vortex merging around the sizes and thresholds at which it goes another way: 256 blobs
(below them the ordered walk alone) and 60 % of the blobs with more than 24 partners
(above it the walk again), with and without the cell grid (4096 blobs).  Bit for bit
against the oracle."""
import numpy as np
import pytest

from dvmpp_b200 import native as N  # noqa: F401  (the fixture's library)
from dvmpp_b200 import workloads as W

pytestmark = pytest.mark.gpu

KEYS = ("x", "z", "circ", "sigma", "u", "w", "uvs", "wvs", "id")


@pytest.mark.parametrize("n", [3, 255, 256, 257, 3000, 5003])
@pytest.mark.parametrize("thr", [2e-6, 1e-5, 3e-5, 6e-5, 1e-4, 1e-3])
def test_routes_give_the_greedy_merge(ctx, port, n, thr):
    rng = np.random.default_rng(n)
    x, z, g, _ = W.wake(n, 3, 0.05)
    d = dict(x=x, z=z, circ=g, sigma=rng.uniform(0.02, 0.05, n), id=np.arange(n, dtype=np.uint32))
    for k in ("u", "w", "uvs", "wvs"):
        d[k] = rng.normal(0, 1, n)
    got, cg = ctx.merge_blobs(d, thr)
    ref, cr = port.merge_blobs(d, thr)
    assert cg == cr
    for k in KEYS:
        assert np.array_equal(got[k], ref[k]), k
