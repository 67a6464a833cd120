"""Host calls whose particles and velocities pass through a stage of at most 2^20 of them:
results in several pieces equal the device calls' bit for bit, and the device memory held
beside the arrays of the call stays that stage.

Bounds: x z circ sigma, u w (self); the same and tx tz, u w per target (at); x z circ sigma
in and out (remesh); 32 MiB of stage, a quarter of it all as room to grow, 1 MiB of
rounding (at: a partial sum per target and 4096 sources besides)."""
import ctypes as C

import numpy as np
import pytest

from dvmpp_b200 import native as N
from dvmpp_b200 import workloads as W

pytestmark = pytest.mark.gpu

MIB = 1 << 20
_u64, _vp, _int = C.c_uint64, C.c_void_p, C.c_int


def _wake(n):
    x, z, g, s = W.wake(n, 7, 0.02)
    return x, z, g, s


def _device(ctx, torch, name, arrays, nout, *tail):
    """Calls a *_device entry point on copies of the arrays; its last two array
    arguments are the results of nout values."""
    d = [None if a is None else torch.from_numpy(a).cuda() for a in arrays]
    out = [torch.empty(nout, dtype=torch.float64, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    f = getattr(ctx.lib, name)
    args = []
    for a in (*d, *out):
        args.append(_vp(a.data_ptr()))
        if len(args) == 4:
            args.append(_u64(arrays[0].size))
        if name.endswith("at_device") and len(args) == 7:
            args.append(_u64(nout))
    rc = f(ctx.h, *args, *(_int(t) for t in tail))
    assert rc == 0
    ctx.sync()
    return [o.cpu().numpy() for o in out]


@pytest.mark.parametrize("n", [1, 1000, MIB, MIB + 1, 3 * MIB + 5])
def test_self(n):
    torch = pytest.importorskip("torch")
    x, z, g, s = _wake(n)
    with N.Context(0) as c:
        u0, w0 = _device(c, torch, "dvm_biot_savart_self_device", (x, z, g, s), n, N.F32)
        before = c.memory()[0]
        u, w = c.biot_savart_self(x, z, g, s, N.F32)
        assert np.array_equal(u, u0) and np.array_equal(w, w0)
        assert c.memory()[0] - before <= 1.25 * (48 * n + 32 * MIB) + MIB


@pytest.mark.parametrize("ns,nt", [(0, 5), (3 * MIB + 5, 300), (5000, 2 * MIB + 3)])
def test_at(ns, nt):
    torch = pytest.importorskip("torch")
    x, z, g, s = _wake(ns) if ns else [np.zeros(0)] * 4
    tx, tz = np.random.default_rng(nt).uniform(-1.0, 1.0, (2, nt))
    with N.Context(0) as c:
        u0, w0 = _device(c, torch, "dvm_biot_savart_at_device", (x, z, g, s, tx, tz), nt, N.F32, 1)
    with N.Context(0) as c:
        before = c.memory()[0]
        u, w = c.biot_savart_at(x, z, g, s, tx, tz, N.F32)
        assert np.array_equal(u, u0) and np.array_equal(w, w0)
        partials = 16 * max(1, -(-ns // 4096)) * (nt + 256)
        assert c.memory()[0] - before <= 1.25 * (32 * (ns + nt) + partials + 32 * MIB) + MIB


@pytest.mark.parametrize("n,out_cap", [(2 * MIB + 7, 3 * MIB), (5000, 2 * MIB + 1), (3 * MIB, 100000)])
def test_remesh(n, out_cap):
    x, z, g, s = _wake(n)
    cells = 250 if out_cap < MIB else 1400
    p = N.RemeshParams(x.min(), x.max(), z.min(), z.max(), (x.max() - x.min()) / cells,
                       (z.max() - z.min()) / cells, 0.02, 0.0, 0)
    with N.Context(0) as c:
        before = c.memory()[0]
        got = c.remesh(x, z, g, s, p, out_cap)
        assert c.memory()[0] - before <= 1.25 * (32 * (n + out_cap) + 32 * MIB) + MIB
    with N.Context(0) as c:
        sim = c.sim(N.Params(capacity=max(n, out_cap), precision=N.F32, ux=1.0), *W.circle(16))
        sim.set_blobs(x, z, g, s)
        sim.remesh(p)
        ref = sim.blobs()
        sim.close()
    assert sum(v.size for v in got) == 4 * ref["x"].size
    for a, k in zip(got, ("x", "z", "circ", "sigma")):
        assert np.array_equal(a, ref[k])


def test_tight_budget():
    """A budget that holds the call's own arrays and their room to grow holds the call."""
    torch = pytest.importorskip("torch")
    n = 300000
    x, z, g, s = _wake(n)
    with N.Context(0) as c:
        u0, w0 = _device(c, torch, "dvm_biot_savart_self_device", (x, z, g, s), n, N.F32)
        used = c.memory()[0]
    with N.Context(0, budget_bytes=used + -(-60 * n // MIB) * MIB) as c:
        u, w = c.biot_savart_self(x, z, g, s, N.F32)
        assert np.array_equal(u, u0) and np.array_equal(w, w0)
