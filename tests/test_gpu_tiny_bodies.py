"""Bodies of up to 16 panels, whose pseudo-inverse goes another way than larger ones', and
the sizes around that: gamma is the least-squares solution, alone and created in a
group with larger bodies.

Tolerance: a stable least-squares solve is off by a modest multiple of cond(A) ulps,
and so is numpy's; 64 cond(A) eps of the largest gamma covers both."""
import numpy as np
import pytest

from dvmpp_b200 import native as N
from dvmpp_b200 import workloads as W

pytestmark = pytest.mark.gpu

SIZES = (3, 4, 9, 15, 16, 17, 18, 24)


def _flat(n):
    t = np.linspace(0.0, 2.0 * np.pi, n + 1)
    x, z = 0.5 * np.cos(t), 5e-3 * np.sin(t)
    x[-1], z[-1] = x[0], z[0]
    return x, z


def _check(sim):
    sim.phase(N.PHASE_SOLVE)
    A, b = sim.influence(), sim.rhs()
    ref = np.linalg.lstsq(A, b, rcond=None)[0]
    s = np.linalg.svd(A, compute_uv=False)
    tol = 64.0 * s[0] / s[-1] * np.finfo(float).eps * np.max(np.abs(ref))
    assert np.max(np.abs(sim.gamma() - ref)) <= tol
    return sim.gamma()


@pytest.mark.parametrize("body", [W.circle, _flat])
def test_gamma(ctx, body):
    p = N.Params(capacity=1024, ux=1.0, uz=0.1)
    bodies = [body(n) for n in SIZES] + [W.circle(200)]
    group = ctx.sims([p] * len(bodies), bodies)
    for b, together in zip(bodies, group):
        alone = ctx.sim(p, *b)
        assert np.array_equal(_check(alone), _check(together))
        alone.close()
        together.close()
