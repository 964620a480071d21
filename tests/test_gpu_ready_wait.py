"""The traversal's bounded wait, driven without a GPU fault.

The internal levels run in one launch; a group waits a bounded number of polls
for its parent's near list and raises PSG_ERR_READY_SPIN instead of waiting for
good.  The lists of the groups that gave up are then whatever an earlier run
left, or never written, so no later kernel may follow them.
PS_B200_OPT_READY_SPIN lowers the limit to a few polls while the first level
publishes ~200 us late, so the waits run out: ps_calc_forces must return
PS_EDEVICE, on a new context as on one that has ticked, and the same context
must then give the bits of a context whose waits never ran out."""

from __future__ import annotations

import re

import numpy as np
import pytest

import polesitter_b200 as P
from polesitter_b200 import workloads as W

pytestmark = pytest.mark.gpu

READY_SPIN = 0x200


def _context(n, theta, cap, order, opts):
    ctx = P.Context(n, theta=theta)
    ctx.set_option(P.OPT_LEAF_CAP, cap)
    if order:
        ctx.set_closure(order)
    for key, value in opts.items():
        ctx.set_option(getattr(P, key), value)
    return ctx


def _gives_up(ctx, p):
    ctx.set_option(P.OPT_READY_SPIN, 4)
    with pytest.raises(P.PolesitterError) as e:
        ctx.tick(p, np.zeros(p.n, np.uint32))
    assert e.value.code == P.PS_EDEVICE
    m = re.search(r"device status error 0x([0-9a-f]+)", str(e.value))
    assert m and int(m.group(1), 16) & READY_SPIN, str(e.value)
    ctx.set_option(P.OPT_READY_SPIN, 0)


@pytest.mark.parametrize("gen,theta,cap,order,opts", [
    (lambda: W.plummer(20000, 31), 2.0, 1, 0, {}),            # sparse leaf pass
    (lambda: W.clumpy_plummer(20000, 32), 2.0, 16, 0, {}),    # merged source leaves
    (lambda: W.clumpy_plummer(20000, 32), 8.0, 1, 0, {}),     # split groups, two launches
    (lambda: W.clumpy_plummer(20000, 32), 6.25, 16, 1, {}),   # ... of order 1
    (lambda: W.clumpy_plummer(20000, 32), 4.0, 1, 0, {"OPT_HEAVY_DEPTH": 3}),
    (lambda: W.clumpy_plummer(20000, 32), 4.0, 1, 0, {"OPT_NEAR_LEVELS": 6}),
    (lambda: W.clumpy_plummer(20000, 32), 3.0, 1, 0, {"OPT_STREAM": 1}),
], ids=["sparse", "merged", "split", "split_order1", "heavy", "chains", "stream"])
def test_ready_wait_runs_out_and_context_recovers(gen, theta, cap, order, opts):
    p0 = gen()
    with _context(p0.n, theta, cap, order, opts) as ctx:
        good = p0.copy()
        ctx.tick(good, np.zeros(good.n, np.uint32))
    small = W.plummer(3000, 33)
    with _context(p0.n, theta, cap, order, opts) as ctx:
        _gives_up(ctx, p0.copy())                 # nothing has been written yet
        for _ in range(2):
            b = p0.copy()
            ctx.tick(b, np.zeros(b.n, np.uint32))
            assert np.array_equal(good.id, b.id)
            for k in ("fx", "fy", "fz"):
                assert np.array_equal(getattr(good, k), getattr(b, k)), k
            _gives_up(ctx, small.copy())          # another tree's lists are there


def test_ready_spin_option_bounds():
    with P.Context(64) as ctx:
        for bad in (-1, 1.5, (1 << 22) + 1):
            with pytest.raises(P.PolesitterError) as e:
                ctx.set_option(P.OPT_READY_SPIN, bad)
            assert e.value.code == P.PS_EINVAL


def test_ensemble_rerun_that_gives_up_is_an_error():
    """A batch tick whose stores have to grow, and whose rerun then gives up: an
    error, not void forces; the next tick is right."""
    torch = pytest.importorskip("torch")
    counts, theta = [20000, 3000], np.array([6.0, 2.0], np.float32)
    heavy = [W.clumpy_plummer(counts[0], 34), W.plummer(counts[1], 35)]
    keys = ("x", "y", "z", "mass")
    n = sum(counts)

    def light():
        out = {k: np.concatenate([getattr(p, k) for p in heavy]) for k in keys}
        for k in ("x", "y", "z"):  # near lists of a few entries
            out[k] = np.zeros(n, np.float32)
            out[k][[1, counts[0] + 1]] = 1.0
        return out

    def full():
        return {k: np.concatenate([getattr(p, k) for p in heavy]) for k in keys}

    class D:
        pass

    def arrays():
        d = D()
        for k in keys + ("fx", "fy", "fz"):
            setattr(d, k, torch.zeros(n, device="cuda"))
        d.id = torch.zeros(n, dtype=torch.int32, device="cuda")
        return d, torch.zeros(n, dtype=torch.int32, device="cuda"), \
            [torch.zeros(n, device="cuda") for _ in range(3)]

    def load(d, v, src):
        for k in keys:
            getattr(d, k).copy_(torch.from_numpy(src[k]))
        for a in v:
            a.zero_()
        torch.cuda.synchronize()

    d, codes, v = arrays()
    with P.Ensemble(counts, theta) as ens:
        load(d, v, full())
        ens.run(d, codes, *v, 1e-3, 1)
        want = {k: getattr(d, k).clone() for k in ("x", "fx", "fy", "fz", "id")}
    d, codes, v = arrays()
    with P.Ensemble(counts, theta) as ens:
        for _ in range(2):
            load(d, v, light())
            ens.run(d, codes, *v, 1e-3, 1)
        ens.set_option(P.OPT_READY_SPIN, 4)
        load(d, v, full())
        with pytest.raises(P.PolesitterError) as e:
            ens.run(d, codes, *v, 1e-3, 1)
        assert e.value.code == P.PS_EDEVICE
        m = re.search(r"device status 0x([0-9a-f]+)", str(e.value))
        assert m and int(m.group(1), 16) & READY_SPIN, str(e.value)
        ens.set_option(P.OPT_READY_SPIN, 0)
        load(d, v, full())
        ens.run(d, codes, *v, 1e-3, 1)
        torch.cuda.synchronize()
        for k, w in want.items():
            assert torch.equal(getattr(d, k), w), k
        with pytest.raises(P.PolesitterError):
            ens.set_option(P.OPT_SORT_SPIN, 1)
