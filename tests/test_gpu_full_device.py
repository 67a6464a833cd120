"""Calls on a device whose memory is taken.  Setting a simulation's blobs has room of its own
in the simulation's arrays; without scratch beside them it still gives the same
state, and still refuses a non-finite value with the simulation left as it was.
Merging without room for its lists gives the same blobs by the ordered walk."""
import numpy as np
import pytest

from dvmpp_b200 import native as N
from dvmpp_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _fill(torch, spare=96, step=128):
    """Takes the device's free memory in blocks (what other allocators keep unused is
    given back to it on the way) but for spare to spare + step MB."""
    spare, blocks, size = torch.empty(spare << 20, dtype=torch.uint8, device="cuda"), [], 32 << 30
    while size >= step << 20:
        try:
            blocks.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
        except torch.OutOfMemoryError:
            size //= 2
    del spare
    torch.cuda.empty_cache()
    return blocks


def test_set_blobs_without_scratch():
    torch = pytest.importorskip("torch")
    n = 1 << 23  # 256 MB of blobs
    rng = np.random.default_rng(5)
    sets = [[rng.normal(0.0, 1.0, n), rng.normal(0.0, 1.0, n), rng.normal(0.0, 1e-3, n), rng.uniform(0.01, 0.02, n)]
            for _ in range(2)]
    with N.Context(0) as c:
        sim = c.sim(N.Params(capacity=n, precision=N.F32, ux=1.0), *W.circle(16))
        try:
            small = [v[:10] for v in sets[0]]
            sim.set_blobs(*small)  # (the code is on the device)
            blocks = _fill(torch)
            try:
                with pytest.raises(torch.OutOfMemoryError):
                    torch.empty(256 << 20, dtype=torch.uint8, device="cuda")
                sim.set_blobs(*sets[0])
                got = sim.blobs()
                assert sim.n == n
                for k, v in zip(("x", "z", "circ", "sigma"), sets[0]):
                    assert np.array_equal(got[k], v)
                for k in ("u", "w", "uvs", "wvs"):
                    assert not np.any(got[k])
                assert np.array_equal(got["id"], np.arange(n))
                bad = [v.copy() for v in sets[1]]
                bad[2][n - 3] = np.inf
                with pytest.raises(N.DvmError, match=f"blob {n - 3}"):
                    sim.set_blobs(*bad)
                assert sim.n == n and np.array_equal(sim.blobs()["circ"], sets[0][2])
                sim.set_blobs(*sets[1])
                assert np.array_equal(sim.blobs()["x"], sets[1][0])
            finally:
                del blocks
                torch.cuda.empty_cache()
        finally:
            sim.close()


def test_merge_without_room_for_lists():
    """3 million blobs: 900 MB with the lists, 450 without; 480 to 608 MB left."""
    torch = pytest.importorskip("torch")
    n = 3_000_000
    x, z, g, s = W.wake(n, 9, 0.02)
    rng = np.random.default_rng(9)
    for a in (x, z):
        a[100:n:500] = a[99:n - 1:500]  # some share a place, which is all that merges
    x[100:n:500] += 1e-12 * rng.normal(size=x[100:n:500].size)
    threshold = 1e-13
    with N.Context(0) as c:
        sim = c.sim(N.Params(capacity=n, precision=N.F32, ux=1.0), *W.circle(16))
        try:
            got = []
            for full in (False, True):
                sim.set_blobs(x, z, g, s)
                blocks = _fill(torch, 480, 128) if full else []
                try:
                    count = sim.merge(threshold)
                finally:
                    del blocks
                    torch.cuda.empty_cache()
                got.append((count, sim.blobs()))
            assert got[0][0] == got[1][0] >= 1000
            for k in got[0][1]:
                assert np.array_equal(got[0][1][k], got[1][1][k])
        finally:
            sim.close()


def test_a_refusal_leaves_nothing_behind():
    """A call that does not fit fails with DVM_ERR_OOM; the next one, which does, is as ever."""
    torch = pytest.importorskip("torch")
    n = 1 << 23
    x, z, g, s = W.wake(1000, 3, 0.05)
    big = [np.zeros(n)] * 4
    mesh = N.RemeshParams(-1.0, 22.0, -5.0, 5.0, 0.0025, 0.0025, 0.05, 0.0, 0)  # 37 million nodes
    with N.Context(0) as c:
        u0, w0 = c.biot_savart_self(x, z, g, s, N.F32)
        c.remesh(x, z, g, s, N.RemeshParams(-1.0, 22.0, -5.0, 5.0, 0.5, 0.5, 0.05, 0.0, 0))
        blocks = _fill(torch)
        try:
            for refused in (lambda: c.biot_savart_self(*big, N.F32), lambda: c.remesh(x, z, g, s, mesh, 1000),
                            lambda: c.merge_blobs(dict(x=big[0], z=big[0], circ=big[0], sigma=big[0], u=big[0], w=big[0],
                                                       uvs=big[0], wvs=big[0]), 1e-9)):
                with pytest.raises(N.DvmError, match=r"^\[2\]"):
                    refused()
                u, w = c.biot_savart_self(x, z, g, s, N.F32)
                assert np.array_equal(u, u0) and np.array_equal(w, w0)
        finally:
            del blocks
            torch.cuda.empty_cache()
