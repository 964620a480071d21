"""Ticks on a device whose memory is nearly full: a store that cannot be grown
must cost speed, not the tick.  The rest of the memory is taken by one plain
allocation; nothing is ever launched on it."""

from __future__ import annotations

import numpy as np
import pytest

import polesitter_b200 as P
from conftest import rel_l2
from polesitter_b200 import workloads as W

pytestmark = pytest.mark.gpu

# FP32 sums of a few thousand terms in another order; the parity tests' bar
FORCE_REL_L2 = 1e-5
MIB = 1 << 20


def _fill(torch, leave):
    """Tensors that take all device memory but `leave` bytes."""
    held = []
    torch.cuda.empty_cache()
    while True:
        free = torch.cuda.mem_get_info()[0] - leave
        if free < 4 * MIB:
            return held
        try:
            held.append(torch.empty(free // (2 * MIB) * 2 * MIB, dtype=torch.uint8,
                                    device="cuda"))
        except torch.cuda.OutOfMemoryError:
            return held


def _forces(p):
    return np.stack([p.fx, p.fy, p.fz], 1).astype(np.float64)


def test_p2p_is_streamed_when_its_records_do_not_fit():
    torch = pytest.importorskip("torch")
    n, theta, cap = 1 << 20, 12.0, 64
    p0 = W.clumpy_plummer(n, 42)
    want, streamed = p0.copy(), p0.copy()
    with P.Context(n, theta=theta) as ctx:
        ctx.set_option(P.OPT_LEAF_CAP, cap)
        ctx.tick(want, np.zeros(n, np.uint32))
        st = ctx.stats()
        assert st["streamed"] == 0 and st["traversal_runs"] > 1  # (the records grew)
        # (the streamed kernels are loaded while there is room)
        ctx.set_option(P.OPT_STREAM, 1)
        ctx.tick(streamed, np.zeros(n, np.uint32))
    with P.Context(n, theta=2.99) as ctx:
        # the near lists and the P2P chunks grow to what the next tick needs,
        # the records do not: no source list is long enough to be segmented
        ctx.tick(p0.copy(), np.zeros(n, np.uint32))
        ctx.set_option(P.OPT_THETA, theta)
        ctx.set_option(P.OPT_LEAF_CAP, cap)
        held = _fill(torch, 24 * MIB)
        got = p0.copy()
        ctx.tick(got, np.zeros(n, np.uint32))
        st = ctx.stats()
        del held
        torch.cuda.empty_cache()
        assert st["near_levels"] == 10 and st["streamed"] == 1
        # with room again, and the choice reset, the records come back
        ctx.set_option(P.OPT_LEAF_CAP, cap)
        again = p0.copy()
        ctx.tick(again, np.zeros(n, np.uint32))
        assert ctx.stats()["streamed"] == 0
    assert np.array_equal(got.id, want.id)
    assert rel_l2(_forces(got), _forces(want)) < FORCE_REL_L2
    assert np.array_equal(_forces(got), _forces(streamed))
    assert np.array_equal(_forces(again), _forces(want))


def test_batch_runs_without_room_for_its_split_groups():
    torch = pytest.importorskip("torch")
    # theta 3 splits the groups above depth 3 of every system: 714 MiB in all
    counts = [520] * 2000
    n = sum(counts)
    p0 = W.uniform_cube(n, 44)

    class D:
        pass

    def run(ens):
        d = D()
        for k in ("x", "y", "z", "mass", "fx", "fy", "fz"):
            setattr(d, k, torch.from_numpy(getattr(p0, k).copy()).cuda())
        d.id = torch.from_numpy(p0.id.view(np.int32).copy()).cuda()
        v = [torch.zeros(n, device="cuda") for _ in range(3)]
        codes = torch.zeros(n, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        ens.run(d, codes, *v, 1e-3, 1)
        torch.cuda.synchronize()
        return d.id.cpu().numpy(), np.stack([a.cpu().numpy() for a in (d.fx, d.fy, d.fz)],
                                            1).astype(np.float64)

    with P.Ensemble(counts, np.full(2000, 3.0, np.float32)) as ens:
        want_id, want = run(ens)
    free = torch.cuda.mem_get_info()[0]
    with P.Ensemble(counts, np.full(2000, 2.0, np.float32)):  # (no split groups)
        need = free - torch.cuda.mem_get_info()[0]
    held = _fill(torch, need + 320 * MIB)
    with P.Ensemble(counts, np.full(2000, 3.0, np.float32)) as ens:
        got_id, got = run(ens)
        del held
        torch.cuda.empty_cache()
        ens.set_leaf_caps(np.full(2000, 1, np.uint32))  # (looks again)
        again_id, again = run(ens)
    assert np.array_equal(got_id, want_id)
    assert rel_l2(got, want) < FORCE_REL_L2
    assert np.array_equal(again_id, want_id) and np.array_equal(again, want)


def test_shallow_leaf_frontiers_come_with_their_first_use():
    torch = pytest.importorskip("torch")
    n = 1 << 20
    frontiers = 64 * 3 * (n // 4 + 4096) * 4
    p0 = W.plummer(n, 45)

    def tick(ctx):
        p = p0.copy()
        ctx.tick(p, np.zeros(n, np.uint32))
        return _forces(p)

    with P.Context(n, theta=2.0) as ctx:
        plain = tick(ctx)
        free = torch.cuda.mem_get_info()[0]
        ctx.set_option(P.OPT_HEAVY_DEPTH, 3)
        want = tick(ctx)
        assert free - torch.cuda.mem_get_info()[0] >= frontiers
    with P.Context(n, theta=2.0) as ctx:
        tick(ctx)
        ctx.set_option(P.OPT_HEAVY_DEPTH, 3)
        held = _fill(torch, 24 * MIB)
        got = tick(ctx)
        del held
        torch.cuda.empty_cache()
        again = tick(ctx)
    assert np.array_equal(got, plain)  # the leaf pass has taken them
    assert rel_l2(got, want) < FORCE_REL_L2
    assert np.array_equal(again, want)
