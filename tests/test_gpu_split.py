"""Leaf groups whose walk is shared out over several warps (the shallow depths
at theta >= 3) and P2P source lists recorded in several segments: the
interaction set equals the oracle's, forces agree to the parity bar, and a
system gives the same bits alone and in a batch."""

from __future__ import annotations

import numpy as np
import pytest

import polesitter_b200 as P
from conftest import rel_l2
from polesitter_b200 import workloads as W

pytestmark = pytest.mark.gpu

# FP32 sums of a few thousand terms in another order; the parity tests' bar
FORCE_REL_L2 = 1e-5


def _far_pair(n, seed):
    """Two tight balls far apart: leaves right below the root."""
    p = W.plummer(n, seed, a=0.01)
    p.x[: n // 3] += np.float32(50.0)
    p.x[0], p.y[0], p.z[0] = -50.0, 40.0, 40.0  # a lone particle: a leaf at depth 1
    return p


def _offset_grid(n, seed):
    """A tiny system at a large offset, where node centres round together and a
    target can be separated from the root itself."""
    p = W.uniform_cube(n, seed)
    for k in ("x", "y", "z"):
        a = getattr(p, k)
        a[:] = np.float32(4096.0) + np.float32(0.002) * a
    return p


@pytest.mark.parametrize("make,theta,cap,order", [
    (lambda: W.clumpy_plummer(3000, 5), 3.0, 1, 0),
    (lambda: W.clumpy_plummer(20000, 6), 3.99, 1, 0),
    (lambda: W.clumpy_plummer(20000, 6), 12.0, 1, 0),     # lists of many segments
    (lambda: W.clumpy_plummer(20001, 7), 6.25, 16, 1),
    (lambda: W.clumpy_plummer(20001, 7), 6.25, 33, 0),    # targets past one record
    (lambda: _far_pair(4097, 8), 4.0, 1, 0),
    (lambda: _far_pair(4097, 8), 6.25, 16, 1),
    (lambda: _offset_grid(4099, 9), 3.0, 1, 0),
    (lambda: W.uniform_cube(9, 10), 8.0, 1, 0),
    (lambda: W.uniform_cube(65, 11), 5.0, 1, 1),
], ids=["t3", "t4", "t12", "order1", "cap33", "far", "far_order1", "offset", "tiny", "small"])
def test_split_groups_match_oracle(oracle, make, theta, cap, order):
    a, b = make(), make()
    # (accum_mode 1: the reference's scalar formula for every source; its vector
    # path's 12-bit rsqrt is itself 2.8e-5 from it on the two tight balls)
    ro = oracle.tick(a, theta=theta, leaf_cap=cap, order=order, accum_mode=1)
    with P.Context(b.n, theta=theta) as ctx:
        ctx.set_option(P.OPT_DEBUG, 1)
        ctx.set_option(P.OPT_LEAF_CAP, cap)
        if order:
            ctx.set_closure(order)
        ctx.set_option(P.OPT_SHRINK_STORES, 1)  # a void first run must leave nothing behind
        codes = np.zeros(b.n, np.uint32)
        ctx.tick(b, codes)
        t, st = ctx.tree(), ctx.stats()
    assert np.array_equal(b.id, a.id)
    assert np.array_equal(t["m2l_cnt"], ro["tree"]["m2l_cnt"])
    assert np.array_equal(t["p2p_cnt"], ro["tree"]["p2p_cnt"])
    assert st["m2l_pairs"] == ro["stats"]["m2l_pairs"]
    assert st["p2p_pairs"] == ro["stats"]["p2p_pairs"]
    assert st["p2p_interactions"] == ro["stats"]["p2p_interactions"]
    F = np.stack([b.fx, b.fy, b.fz], 1).astype(np.float64)
    G = np.stack([a.fx, a.fy, a.fz], 1).astype(np.float64)
    assert rel_l2(F, G) < FORCE_REL_L2
    if not order:
        assert rel_l2(t["local_exp"], ro["tree"]["l_tot"]) < FORCE_REL_L2


def test_split_groups_in_a_batch_equal_alone():
    torch = pytest.importorskip("torch")
    parts = [W.clumpy_plummer(9001, 1), W.uniform_cube(4097, 2), W.clumpy_plummer(20011, 3)]
    theta, caps = np.array([6.0, 2.0, 3.5], np.float32), np.array([16, 1, 4], np.uint32)
    counts = [p.n for p in parts]
    offs = np.concatenate([[0], np.cumsum(counts)])

    class D:
        pass

    d = D()
    for k in ("x", "y", "z", "mass", "fx", "fy", "fz"):
        setattr(d, k, torch.from_numpy(np.concatenate([getattr(p, k) for p in parts])).cuda())
    d.id = torch.from_numpy(np.concatenate([p.id for p in parts]).view(np.int32)).cuda()
    v = [torch.zeros(offs[-1], device="cuda") for _ in range(3)]
    codes = torch.zeros(offs[-1], dtype=torch.int32, device="cuda")
    with P.Ensemble(counts, theta) as ens:
        ens.set_leaf_caps(caps)
        ens.run(d, codes, *v, 1e-3, 2)
    torch.cuda.synchronize()
    for k, p in enumerate(parts):
        w = [np.zeros(p.n, np.float32) for _ in range(3)]
        with P.Context(p.n, theta=float(theta[k])) as ctx:
            ctx.set_option(P.OPT_LEAF_CAP, int(caps[k]))
            ctx.run_ticks(p, np.zeros(p.n, np.uint32), *w, 1e-3, 2)
        for key in ("x", "y", "z", "fx", "fy", "fz"):
            got = getattr(d, key)[offs[k]:offs[k + 1]].cpu().numpy()
            assert np.array_equal(got, getattr(p, key)), (k, key)
