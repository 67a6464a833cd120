"""Vortex merging where its parallel chains can go wrong: sizes around the cell
grid's threshold (4096 blobs), blobs that absorb more than a chain holds (16),
chains that lose members to earlier absorbers, and more blobs than the shared
present-bits hold (1 572 864).  Bit for bit against the oracle; the last
against pairs that merge alone, whose result is known."""
import numpy as np
import pytest

from dvmpp_b200 import native as N
from dvmpp_b200 import workloads as W

pytestmark = pytest.mark.gpu

KEYS = ("x", "z", "circ", "sigma", "u", "w", "uvs", "wvs")


def _set(kind, n, seed):
    rng = np.random.default_rng(seed)
    x, z, g, s = W.wake(n, seed, 0.08)
    if kind == "one sign":  # every blob has many takers: long, overlapping chains
        x, z, g = rng.uniform(0, 1, n), rng.uniform(0, 1, n), rng.uniform(1e-4, 1e-3, n)
    elif kind == "tiny":  # small circulations reach far: full scans
        g = g * 10.0 ** rng.uniform(-9, 0, n)
    d = dict(x=x, z=z, circ=g, sigma=rng.uniform(0.02, 0.05, n), id=np.arange(n, dtype=np.uint32))
    for k in ("u", "w", "uvs", "wvs"):
        d[k] = rng.normal(0, 1, n)
    return d


@pytest.mark.parametrize("kind,n,thr", [
    ("wake", 2, 1.0), ("wake", 4095, 2e-6), ("wake", 4096, 2e-6), ("wake", 12000, 2e-6),
    ("wake", 8000, 2e-4), ("one sign", 6000, 2e-5), ("tiny", 6000, 2e-6), ("tiny", 3000, 1.0)])
def test_chains_give_the_greedy_merge(ctx, port, kind, n, thr):
    d = _set(kind, n, n)
    got, cg = ctx.merge_blobs(d, thr)
    ref, cr = port.merge_blobs(d, thr)
    assert cg == cr
    for k in KEYS + ("id",):
        assert np.array_equal(got[k], ref[k]), k


def test_more_blobs_than_shared_bits(ctx):
    pairs = 800_000
    side = int(np.ceil(np.sqrt(pairs)))
    rng = np.random.default_rng(1)
    cx, cz = (np.arange(pairs) % side).astype(float), (np.arange(pairs) // side).astype(float)
    order = rng.permutation(2 * pairs)
    x, z = np.concatenate([cx, cx + 2.0 ** -14])[order], np.concatenate([cz, cz])[order]
    one = np.ones(2 * pairs)
    d = dict(x=x, z=z, circ=one, sigma=0.5 * one, u=one, w=one, uvs=one, wvs=one)
    got, count = ctx.merge_blobs(d, 1e-3)
    assert count == pairs and got["x"].size == pairs
    first = np.sort(np.stack([np.argsort(order)[:pairs], np.argsort(order)[pairs:]]), axis=0)[0]
    at = np.argsort(first)  # surviving blobs keep the earlier index's place
    assert np.array_equal(got["x"], (cx + 2.0 ** -15)[at]) and np.array_equal(got["z"], cz[at])
    assert np.all(got["circ"] == 2.0) and np.all(got["sigma"] == 0.5) and np.all(got["u"] == 0.0)
