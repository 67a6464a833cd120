"""A solve or a sheet velocity called alone where the blobs' count decides how it sums:
simulations with far more room than blobs, panel counts around the rules' lines
(128, 256, 512, 640 panels), and more panels than one staged set (128).  FP32 against FP64 to
the FP32 path's 1e-5 relative L2, and the same bits whatever the room where both sum pairs.
The sheet velocity's bar is that and, for each blob, 4 x 2^-24 sqrt(np) max |gamma| for the
order-one terms that cancel in far panels' closed forms (one far blob alone has little
else: its velocity is a small remainder of them)."""
import numpy as np
import pytest

from dvmpp_b200 import native as N
from dvmpp_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _lone(ctx, prec, cap, bx, bz, blobs):
    sim = ctx.sim(N.Params(capacity=cap, precision=prec, ux=1.0, uz=0.3), bx, bz)
    sim.set_blobs(*blobs)
    sim.phase(N.PHASE_SOLVE)
    sim.phase(N.PHASE_SHEETBC)
    d = sim.blobs()
    out = sim.gamma(), sim.rhs(), d["uvs"], d["wvs"]
    sim.close()
    return out


@pytest.mark.parametrize("npan", [3, 127, 128, 129, 256, 257, 512, 513, 640, 641, 2047])
@pytest.mark.parametrize("n,cap", [(1, 1024), (257, 1 << 20), (5000, 1 << 20), (150000, 1 << 20)])
def test_lone_phases_with_room(ctx, npan, n, cap):
    bx, bz = W.circle(npan)
    blobs = W.wake(n, npan, 0.03)
    got, ref = _lone(ctx, N.F32, cap, bx, bz, blobs), _lone(ctx, N.F64, max(n, 1024), bx, bz, blobs)
    closed = 4.0 * 2.0 ** -24 * np.sqrt(npan * n) * np.max(np.abs(ref[0]))
    for a, b, rounding in zip(got, ref, (0.0, 0.0, closed, closed)):
        assert np.all(np.isfinite(a))
        assert np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(b) + rounding


@pytest.mark.parametrize("npan", [128, 200, 640])
def test_sheet_velocity_does_not_depend_on_the_room(ctx, npan):
    bx, bz = W.circle(npan)
    blobs = W.wake(5000, npan, 0.03)
    gamma = np.cos(np.linspace(0.0, 6.0, npan))
    got = []
    for cap in (5000, 1 << 20):
        sim = ctx.sim(N.Params(capacity=cap, precision=N.F32, ux=1.0), bx, bz)
        sim.set_blobs(*blobs)
        sim.set_gamma(gamma)
        sim.phase(N.PHASE_SHEETBC)
        got.append(sim.blobs())
        sim.close()
    assert np.array_equal(got[0]["uvs"], got[1]["uvs"]) and np.array_equal(got[0]["wvs"], got[1]["wvs"])
