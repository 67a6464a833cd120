"""Reserving a context's workspace: a batch that it was reserved for finds it large
enough, so its first step takes no memory more (and would neither wait nor drop
captured graphs for it).  FP64 simulations, whose partial sums depend on the capacity
in steps, alone and together."""
import numpy as np
import pytest

from dvmpp_b200 import native as N
from dvmpp_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("caps", [[1024], [8192], [9000], [20000], [65536], [131072], [262144], [1 << 20], [3 << 20],
                                  [1024] * 20, [9000] * 9, [65536] * 3, [500, 65536, 131072, 40000]])
def test_first_step_after_reserve(caps):
    with N.Context(0) as c:
        bx, bz = W.circle(32)
        c.reserve(sum(caps), len(caps), 32, with_delete=True)
        sims = []
        for k, cap in enumerate(caps):
            sims.append(c.sim(N.Params(capacity=cap, precision=N.F64, ux=1.0, dt=0.02), bx, bz))
            x, z, g, s = W.wake(100, k, 0.05)
            sims[-1].set_blobs(x, z, g, s)
        before = c.memory()[0]
        c.step_batch(sims, 1)
        assert c.memory()[0] == before
        for s in sims:
            s.close()


def test_server_reserves_one_set_up():
    """A server's run holds device memory for its workspace, the largest simulations and one
    body's set-up scratch (about 32 np^2 bytes), with 48 MB for the pool's
    granularity and a context's own tables."""
    torch = pytest.importorskip("torch")
    npan = 2047

    def run(c, panels):
        srv = N.Server(c)
        p = N.Params(capacity=1024 + 4 * panels, precision=N.F32, rng=N.RNG_PHILOX, ux=1.0, dt=0.02)
        srv.submit(p, *W.circle(panels), 1)
        srv.run()
        assert srv.stats()["completed"] == 1
        srv.close()
        return N.sim_bytes(p, panels)

    with N.Context(0) as c:
        run(c, 300)  # (code on the device)
    with N.Context(0) as c:
        free0 = torch.cuda.mem_get_info()[0]
        slab = run(c, npan)
        taken = free0 - torch.cuda.mem_get_info()[0]
        ws = N.C.c_uint64()
        assert c.lib.dvm_ctx_workspace_bytes(c.h, N.C.byref(ws)) == 0
        m = npan + 1
        work = 8 * (2 * npan * npan + m * (npan + m) + 2 * m + 2 * npan + 8)
        assert taken <= ws.value + slab + work + 48 * (1 << 20)


def test_a_refused_workspace_leaves_the_old_one():
    """A reservation that the budget does not hold, and a call on the workspace after it."""
    x, z, g, s = W.wake(5000, 3, 0.05)
    with N.Context(0, budget_bytes=200 << 20) as c:
        u0, w0 = c.biot_savart_self(x, z, g, s, N.F32)
        held = c.memory()[0]
        with pytest.raises(N.DvmError, match=r"^\[2\]"):
            c.reserve(1 << 26, 4, 64)
        assert c.memory()[0] == held
        u, w = c.biot_savart_self(x, z, g, s, N.F32)
        assert np.array_equal(u, u0) and np.array_equal(w, w0)
