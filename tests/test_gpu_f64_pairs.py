"""FP64 blob-on-blob sums where the reciprocal's range and the chunking can go
wrong: scales at which r^2 leaves the iteration's range (IEEE takes over), and
counts around a tile (256), a chunk (64) and a chunk's part of a tile.  Against
the oracle to 1e-12 of the field, the FP64 path's bar."""
import numpy as np
import pytest

from dvmpp_b200 import native as N
from dvmpp_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,scale", [(600, 1e-148), (600, 1e-60), (600, 1e60), (600, 1e147),
                                     (63, 1.0), (64, 1.0), (65, 1.0), (511, 1.0), (513, 1.0),
                                     (6001, 1.0), (20000, 1.0)])
def test_f64_pairs_at_any_scale(ctx, port, n, scale):
    x, z, g, s = W.wake(n, n, 0.05)
    x, z, s = x * scale, z * scale, s * scale
    u0, w0 = port.direct_self(x, z, g, s)
    u, w = ctx.biot_savart_self(x, z, g, s, N.F64)
    ref = max(np.max(np.abs(u0)), np.max(np.abs(w0)))
    assert np.max(np.abs(u - u0)) <= 1e-12 * ref and np.max(np.abs(w - w0)) <= 1e-12 * ref
