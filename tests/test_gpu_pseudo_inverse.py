"""Pseudo-inverse of the influence matrix: every way a body can take.

Which way depends on the residual of the first approximation, so on how nearly
singular the matrix is: one step (circles, ellipses), one step and a projection
(airfoils), repeated steps and a projection (thin airfoils), a Householder
factorisation (plates).  Tile edges of 32 panels in each.

Tolerance: a stable least-squares solve is off by a modest multiple of cond(A) ulps,
and so is numpy's; 64 cond(A) eps of the largest gamma covers both.
"""
import numpy as np
import pytest

from dvmpp_b200 import native as N
from dvmpp_b200 import workloads as W

pytestmark = pytest.mark.gpu


def params():
    p = N.Params(capacity=16384, rng_capacity=1 << 20)
    p.ux, p.uz = 1.0, 0.1
    return p


BODIES = (
    [W.circle(n) for n in (3, 31, 32, 33, 64, 65)]
    + [W.ellipse(n, a=0.5, b=0.1, incidence_deg=11) for n in (97, 512, 513)]
    + [W.joukowski(n, thickness=0.12, aoa_deg=5) for n in (40, 96, 200)]  # projection
    + [W.joukowski(n, thickness=0.002, aoa_deg=4) for n in (60, 129)]  # repeated
    + [W.joukowski(n, thickness=1e-5, aoa_deg=3) for n in (50, 300, 700, 1100)]  # Householder
)


@pytest.mark.parametrize("body", BODIES, ids=lambda b: str(len(b[0]) - 1))
def test_gamma_is_the_least_squares_solution(ctx, body):
    s = ctx.sim(params(), *body)
    s.phase(N.PHASE_SOLVE)
    A, b = s.influence(), s.rhs()
    ref = np.linalg.lstsq(A, b, rcond=None)[0]
    tol = 64 * np.linalg.cond(A) * np.finfo(float).eps
    assert np.max(np.abs(s.gamma() - ref)) <= tol * np.max(np.abs(ref))
    s.close()


def test_group_of_every_way_equals_alone(ctx):
    """More bodies than one group holds, and members that leave it at each stage."""
    bodies = [b for b in BODIES if len(b[0]) - 1 < 250]
    group = ctx.sims([params()] * len(bodies), bodies)
    for g, body in zip(group, bodies):
        alone = ctx.sim(params(), *body)
        assert g.save() == alone.save(), g.np
        alone.close()
        g.close()
