"""P2P source lists with neighbouring leaves merged into one range (leaf
capacities of 8 and more): the interaction set equals the oracle's and the
forces agree to the parity bar on both sides of that capacity, with runs of
siblings, partly wanted sources, leaves past one step of 32 sources and
coincident particles, plain and compensated."""

from __future__ import annotations

import numpy as np
import pytest

import polesitter_b200 as P
from conftest import rel_l2
from polesitter_b200 import workloads as W

pytestmark = pytest.mark.gpu

# FP32 sums of a few thousand terms in another order; the parity tests' bar
FORCE_REL_L2 = 1e-5


def _stacked(n, seed):
    """Coincident particles: deepest-level leaves far above the capacity."""
    p = W.clumpy_plummer(n, seed)
    for k in ("x", "y", "z"):
        a = getattr(p, k)
        a[100:170] = a[100]
        a[500:533] = a[500]
    return p


@pytest.mark.parametrize("make", [
    lambda: W.clumpy_plummer(6001, 21),
    lambda: W.uniform_cube(4096, 22),
    lambda: _stacked(5003, 23),
], ids=["clumpy", "cube", "stacked"])
@pytest.mark.parametrize("theta,cap,order,kahan", [
    (1.0, 7, 0, 0), (1.0, 8, 0, 0), (2.5, 9, 0, 1), (6.25, 8, 1, 0), (4.0, 70, 0, 0),
])
def test_merged_source_leaves_match_oracle(oracle, make, theta, cap, order, kahan):
    a, b = make(), make()
    ro = oracle.tick(a, theta=theta, leaf_cap=cap, order=order, accum_mode=1)
    with P.Context(b.n, theta=theta) as ctx:
        ctx.set_option(P.OPT_DEBUG, 1)
        ctx.set_option(P.OPT_LEAF_CAP, cap)
        ctx.set_option(P.OPT_KAHAN, kahan)
        if order:
            ctx.set_closure(order)
        ctx.tick(b, np.zeros(b.n, np.uint32))
        t, st = ctx.tree(), ctx.stats()
    assert np.array_equal(b.id, a.id)
    assert np.array_equal(t["p2p_cnt"], ro["tree"]["p2p_cnt"])
    assert st["p2p_pairs"] == ro["stats"]["p2p_pairs"]
    assert st["p2p_interactions"] == ro["stats"]["p2p_interactions"]
    F = np.stack([b.fx, b.fy, b.fz], 1).astype(np.float64)
    G = np.stack([a.fx, a.fy, a.fz], 1).astype(np.float64)
    assert rel_l2(F, G) < FORCE_REL_L2


def test_many_short_records_match_streamed_sums():
    """So many full-leaf P2P records that they are loaded ahead: against the
    sums taken in the leaf pass itself."""
    n = 1 << 20
    p = W.clumpy_plummer(n, 24)
    for k in ("x", "y", "z"):
        a = getattr(p, k)
        a[1000:1040] = a[1000]  # one leaf of 40: every group takes the recorded path
    out = []
    for stream in (0, 1):
        b = p.copy()
        with P.Context(n, theta=1.0) as ctx:
            ctx.set_option(P.OPT_DEBUG, 1)
            ctx.set_option(P.OPT_STREAM, stream)
            ctx.tick(b, np.zeros(n, np.uint32))
            out.append((np.stack([b.fx, b.fy, b.fz], 1).astype(np.float64), b.id, ctx.stats()))
    (F, fi, fs), (G, gi, gs) = out
    assert fs["dense_records"] >= 64 * 148 * 16  # from here on they are loaded ahead
    assert fs["p2p_interactions"] == gs["p2p_interactions"]
    assert np.array_equal(fi, gi)
    assert rel_l2(F, G) < FORCE_REL_L2
