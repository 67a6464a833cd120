"""Host calls at the sizes where they go another way: up to 512 particles, points or blobs
are packed and converted on the host, and up to 8192 blobs one block finds the sort's
domain.  The same bits as the device calls and as larger calls' parts; a set with a
non-finite value leaves the simulation as it was either way."""
import ctypes as C

import numpy as np
import pytest

from dvmpp_b200 import native as N
from dvmpp_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _on_device(ctx, torch, prec, x, z, g, s):
    d = [torch.from_numpy(np.array(a)).cuda() for a in (x, z, g, s, x, x)]
    torch.cuda.synchronize()
    p = [C.c_void_p(t.data_ptr()) for t in d]
    assert ctx.lib.dvm_biot_savart_self_device(ctx.h, *p[:4], x.size, *p[4:], prec) == 0
    ctx.sync()
    return [t.cpu().numpy() for t in d[4:]]


@pytest.mark.parametrize("prec", [N.F32, N.F64])
@pytest.mark.parametrize("n", [1, 2, 511, 512, 513, 8192, 8193])
def test_self(ctx, port, n, prec):
    torch = pytest.importorskip("torch")
    x, z, g, s = W.wake(n, n, 0.05)
    u, w = ctx.biot_savart_self(x, z, g, s, prec)
    u0, w0 = _on_device(ctx, torch, prec, x, z, g, s)
    assert np.array_equal(u, u0) and np.array_equal(w, w0)
    ru, rw = port.direct_self(x, z, g, s)
    tol = 1e-5 if prec == N.F32 else 1e-12
    assert np.linalg.norm(u - ru) <= tol * np.linalg.norm(ru) + 1e-300
    assert np.linalg.norm(w - rw) <= tol * np.linalg.norm(rw) + 1e-300


def test_domain_of_part_finite_positions(ctx):
    """A non-finite position leaves no mark on the domain: the others' box is as without it, so
    the blobs far from it keep their order, and the call returns."""
    x, z, g, s = W.wake(600, 3, 0.05)
    for bad in (np.nan, np.inf, -np.inf):
        b = x.copy()
        b[17] = bad
        u, _ = ctx.biot_savart_self(b, z, g, s, N.F64)
        assert u.shape == x.shape
    u, w = ctx.biot_savart_self(np.full(5, 2.0), np.full(5, -1.0), g[:5], s[:5], N.F32)  # one place
    assert np.all(u == 0.0) and np.all(w == 0.0)


@pytest.mark.parametrize("ns,nt", [(512, 512), (513, 512), (512, 513), (3, 1), (0, 7), (5000, 512)])
def test_at_is_its_parts(ctx, ns, nt):
    x, z, g, s = W.wake(ns, 5, 0.05) if ns else [np.zeros(0)] * 4
    tx, tz = np.random.default_rng(nt).uniform(-1.0, 5.0, (2, nt + 700))
    u, w = ctx.biot_savart_at(x, z, g, s, tx[:nt], tz[:nt], N.F64)
    ru, rw = ctx.biot_savart_at(x, z, g, s, tx, tz, N.F64)
    tol = 1e-12 * max(np.max(np.abs(ru)), np.max(np.abs(rw))) + 1e-300
    assert np.max(np.abs(u - ru[:nt])) <= tol and np.max(np.abs(w - rw[:nt])) <= tol


def test_probe_is_its_parts(ctx):
    bx, bz = W.circle(64)
    sim = ctx.sim(N.Params(capacity=4096, precision=N.F64, ux=1.0, uz=0.2), bx, bz)
    sim.set_blobs(*W.wake(3000, 5, 0.05))
    sim.phase(N.PHASE_SOLVE)
    px, pz = np.random.default_rng(1).uniform(-3.0, 3.0, (2, 1100))
    whole = [np.array(v) for v in sim.probe(px, pz)]
    for n in (1, 512, 513):
        for part, ref in zip(sim.probe(px[:n], pz[:n]), whole):
            assert np.max(np.abs(part - ref[:n])) <= 1e-12 * np.max(np.abs(ref))
    sim.close()


@pytest.mark.parametrize("n", [0, 1, 512, 513])
def test_set_blobs(ctx, n):
    sim = ctx.sim(N.Params(capacity=2048, ux=1.0), *W.circle(16))
    old = W.wake(700, 2, 0.05)
    sim.set_blobs(*old)
    sim.phase(N.PHASE_BIOTSAVART)
    if n:
        for k in range(4):
            bad = [np.array(v[:n]) for v in old]
            bad[k][n - 1] = np.inf
            with pytest.raises(N.DvmError, match=f"blob {n - 1}"):
                sim.set_blobs(*bad)
        assert sim.n == 700 and np.any(sim.blobs()["u"]) and np.array_equal(sim.blobs()["x"], old[0])
    new = [v[:n] for v in W.wake(800, 4, 0.05)]
    sim.set_blobs(*new)
    got = sim.blobs()
    assert sim.n == n and np.array_equal(got["id"], np.arange(n))
    for k, v in zip(("x", "z", "circ", "sigma"), new):
        assert np.array_equal(got[k], v)
    for k in ("u", "w", "uvs", "wvs"):
        assert not np.any(got[k])
    sim.close()
