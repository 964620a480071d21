"""A first tick at a theta so wide that the near lists do not fit: the runs that
only find out what has to grow are short ones.  The last of them is the first to
run k_heavy_leaf, whose frontiers may run out; the leaf pass beside it, most of
such a tick, must not be taken to its end then."""

from __future__ import annotations

import time

import numpy as np
import pytest

import polesitter_b200 as P
from polesitter_b200 import workloads as W

pytestmark = pytest.mark.gpu


def test_first_wide_tick_costs_about_one_run():
    p0 = W.clumpy_plummer(1 << 20, 424242)

    def tick(ctx):
        p = p0.copy()
        t0 = time.perf_counter()
        ctx.tick(p, np.zeros(p.n, np.uint32))
        return time.perf_counter() - t0, np.stack([p.fx, p.fy, p.fz])

    ratios = []
    for _ in range(2):  # (an allocation of gigabytes can take some 0.5 s by itself)
        with P.Context(p0.n, theta=24.0) as ctx:
            first, a = tick(ctx)
            assert ctx.stats()["traversal_runs"] > 1
            again, b = tick(ctx)
            st = ctx.stats()
        assert st["traversal_runs"] == 1 and st["streamed"] == 1
        assert np.array_equal(a, b)
        ratios.append(first / again)
    # the last run twice would be 2; the short ones take 0.1 to 0.2 of a tick
    assert min(ratios) < 1.6, ratios
