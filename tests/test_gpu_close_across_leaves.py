"""FP32 blob-on-blob sums with pairs of blobs that FP32 offsets do not tell apart, the
two of a pair in different leaves of the sorted order, and core sizes below their
distance (zero among them): every velocity stays finite, as in FP64, and the blobs
that have no such neighbour keep the FP32 path's 1e-5 relative L2.

The sort is stable and the two of a pair share a cell of the curve, so an odd blob in the
first cell makes a pair straddle every boundary of 64."""
import numpy as np
import pytest

from dvmpp_b200 import native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sigma", [0.0, 1e-12])
@pytest.mark.parametrize("gap", [1e-10, 1e-30])
@pytest.mark.parametrize("pairs,scale", [(64, 1.0), (3000, 1.0), (3000, 1e-6), (20000, 1e3)])
def test_pairs_astride_leaves(ctx, pairs, scale, gap, sigma):
    rng = np.random.default_rng(pairs)
    n = 2 * pairs + 1
    x, z = np.zeros(n), np.zeros(n)  # blob 0: the curve's first cell
    x[1::2], z[1::2] = rng.uniform(0.05, 1.0, (2, pairs))
    x[2::2], z[2::2] = x[1::2], z[1::2]
    x[1], z[1], x[2], z[2] = 1.0, 1.0, 1.0, 1.0
    x *= scale
    z *= scale
    if gap > 1e-20:
        x[2::2] += gap * scale
    else:  # FP64 cannot hold the gap there either; near the axis it can
        z[1::2] = 0.0
        z[2::2] = gap * scale
    g = rng.normal(0.0, 1e-3, n)
    s = np.full(n, sigma * scale)
    u, w = ctx.biot_savart_self(x, z, g, s, N.F32)
    assert np.all(np.isfinite(u)) and np.all(np.isfinite(w))
    u0, w0 = ctx.biot_savart_self(x, z, g, s, N.F64)
    assert np.all(np.isfinite(u0)) and np.all(np.isfinite(w0))
    assert np.hypot(u[0] - u0[0], w[0] - w0[0]) <= 1e-5 * np.hypot(u0[0], w0[0])
