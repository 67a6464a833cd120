"""FP64 blob-on-blob sums with pairs so close that r^2 is denormal (a reciprocal of it
overflows), inside a core that is far wider, ten times and a thousand times as wide as
their distance, among other blobs.  Against the oracle.

Bound: 1e-12 of the blob's own speed, the FP64 path's bar; where 1 - exp cancels to 1e-4
or less the two exponentials' last bits weigh more: 2^-52 over that."""
import numpy as np
import pytest

from dvmpp_b200 import native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("r,sigma,tol", [(1e-155, 0.05, 1e-12), (3e-160, 0.05, 1e-12), (1e-155, 1e-154, 1e-10),
                                         (1e-155, 1e-153, 1e-11), (5e-155, 1e-152, 1e-9)])
def test_denormal_distance(ctx, port, r, sigma, tol):
    x = np.array([0.0, r, 0.0, 0.31, -0.2, 0.1])
    z = np.array([0.0, 0.0, r, 0.17, 0.4, -0.3])
    g = np.array([1e-3, -2e-3, 1.5e-3, 0.02, -0.01, 0.03])
    s = np.array([sigma, sigma, sigma, 0.05, 0.05, 0.05])
    u0, w0 = port.direct_self(x, z, g, s)
    assert np.all(np.isfinite(u0)) and np.all(np.isfinite(w0))
    u, w = ctx.biot_savart_self(x, z, g, s, N.F64)
    assert np.all(np.hypot(u - u0, w - w0) <= tol * np.hypot(u0, w0))
