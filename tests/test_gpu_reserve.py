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
