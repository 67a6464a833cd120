"""The FP32 blob-on-blob path's far field (expansions over the tree of sorted
blobs, csrc/dvm_tree.cuh) against the all-pairs FP64 path, at the sizes and
layouts where the tree can go wrong: part-filled leaves, one leaf, the size
from which target groups nest (256 leaves), blobs so spread or so dense that a
group takes nodes target by target or sums every leaf pair by pair (its list
then overflows and is worked off in parts), and scales far from 1.

Bound: the FP32 path's bar of 1e-5 relative L2 for velocities.  The FP32 pair
terms stay below it in the all-pairs tests; the expansions add at most
2^-24 / (1 - 1/2) = 1.2e-7 of sum |Gamma| / (2 pi D) per blob.
"""
import numpy as np
import pytest

from dvmpp_b200 import native as N
from dvmpp_b200 import workloads as W

pytestmark = pytest.mark.gpu

REL_L2 = 1e-5


def _layout(name, n, rng):
    if name == "wake":
        x, z, _, _ = W.wake(n, n, 0.05)
    elif name == "fringe":  # a dense core inside a sparse ring ten times wider
        x, z = rng.normal(0.0, 0.3, (2, n))
        k = n // 50
        r, t = rng.uniform(3.0, 10.0, k), rng.uniform(0.0, 2 * np.pi, k)
        x[:k], z[:k] = r * np.cos(t), r * np.sin(t)
    elif name == "clusters":  # two clusters far apart compared with their size
        x, z = rng.normal(0.0, 1e-3, (2, n))
        x[n // 2:] += 40.0
    else:  # blobs along a line
        x, z = np.sort(rng.uniform(-3.0, 3.0, n)), np.zeros(n)
    return x, z


@pytest.mark.parametrize("name,n,sigma,scale", [
    ("wake", 1, 0.05, 1.0), ("wake", 63, 0.05, 1.0), ("wake", 64, 0.05, 1.0),
    ("wake", 65, 0.05, 1.0), ("wake", 255 * 64, 0.05, 1.0), ("wake", 255 * 64 + 1, 0.05, 1.0),
    ("wake", 70001, 0.02, 1.0), ("wake", 9001, 0.05, 1e-9), ("wake", 9001, 0.05, 1e9),
    ("fringe", 30011, 0.02, 1.0), ("clusters", 20011, 1e-4, 1.0), ("line", 20011, 0.01, 1.0),
    ("wake", 40000, 30.0, 1.0),  # every pair inside a core: 625 leaves summed by each
])
def test_far_field_matches_all_pairs(ctx, name, n, sigma, scale):
    rng = np.random.default_rng(n)
    x, z = _layout(name, n, rng)
    g = rng.normal(0.0, 1e-3, n)
    x, z, s = x * scale, z * scale, np.full(n, sigma * scale)
    u0, w0 = ctx.biot_savart_self(x, z, g, s, N.F64)
    u, w = ctx.biot_savart_self(x, z, g, s, N.F32)
    ref = np.sqrt(np.sum(u0 ** 2 + w0 ** 2))
    err = np.sqrt(np.sum((u - u0) ** 2 + (w - w0) ** 2))
    assert err <= REL_L2 * ref, (err, ref)
