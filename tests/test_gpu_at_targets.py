"""At-target velocities where the packed sources, the chunks and the combine can go
wrong: odd counts of sources, targets around a tile (256) and a combine block
(32), many and few chunks, targets on sources, and non-finite sources, which a
skipping call leaves out.  Against the oracle, with the bars of the at-target
tests (FP64 1e-12 of the field, FP32 1e-5 relative L2)."""

import numpy as np
import pytest

from dvmpp_b200 import native as N
from dvmpp_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [N.F64, N.F32])
@pytest.mark.parametrize("ns,nt", [(1, 1), (2, 31), (255, 33), (257, 255), (5001, 257), (40001, 1),
                                   (3, 5000), (20000, 700)])
def test_at_targets(ctx, port, ns, nt, prec):
    x, z, g, s = W.wake(ns, ns, 0.06)
    rng = np.random.default_rng(nt)
    tx, tz = rng.uniform(-1, 12, nt), rng.normal(0, 1, nt)
    k = min(ns, nt, 7)
    tx[:k], tz[:k] = x[:k], z[:k]
    u0, w0 = port.direct_at(x, z, g, s, tx, tz)
    u, w = ctx.biot_savart_at(x, z, g, s, tx, tz, prec)
    if prec == N.F64:
        ref = max(np.max(np.abs(u0)), np.max(np.abs(w0)))
        assert np.max(np.abs(u - u0)) <= 1e-12 * ref and np.max(np.abs(w - w0)) <= 1e-12 * ref
    else:
        ref = np.sqrt(np.sum(u0 ** 2 + w0 ** 2))
        assert np.sqrt(np.sum((u - u0) ** 2 + (w - w0) ** 2)) <= 1e-5 * ref


@pytest.mark.parametrize("prec", [N.F64, N.F32])
def test_nan_sources_are_skipped(ctx, prec):
    x, z, g, s = W.wake(600, 3, 0.06)
    tx, tz = W.collocation_circle(64)
    bad = [x.copy(), z.copy(), g, s]
    bad[0][10], bad[1][301] = np.nan, np.nan
    keep = np.delete(np.arange(600), [10, 301])
    u, w = ctx.biot_savart_at(*bad, tx, tz, prec)
    u0, w0 = ctx.biot_savart_at(x[keep], z[keep], g[keep], s[keep], tx, tz, prec)
    tol = 1e-12 if prec == N.F64 else 1e-5
    assert np.linalg.norm(u - u0) <= tol * np.linalg.norm(u0)
    assert np.linalg.norm(w - w0) <= tol * np.linalg.norm(w0)
