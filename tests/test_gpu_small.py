"""Sizes at the edges of the small-system paths: the one-block sort (up to 4,096
particles, 1,024 threads), the tree build that adds up its tile counts itself
(up to 64 tiles of 1,024), and pageable arrays staged through pinned rows (up
to 32,768 particles)."""

from __future__ import annotations

import numpy as np
import pytest

import polesitter_b200 as P
from conftest import rel_l2
from polesitter_b200 import workloads as W

pytestmark = pytest.mark.gpu

FORCE_REL_L2 = 1e-5  # the parity tests' bar
TOPO = ("depth", "start", "count", "nchild", "octant", "first_child", "parent")


def _particles(n, kind):
    p = W.uniform_cube(n, n + 1)
    if kind == "ties":  # many equal codes: the sort has to be stable
        for k in ("x", "y", "z"):
            a = getattr(p, k)
            a[:] = np.round(a * 4.0) / np.float32(4.0)
    p.id[:] = np.random.default_rng(n).permutation(n).astype(np.uint32)
    return p


@pytest.mark.parametrize("kind", ["uniform", "ties"])
@pytest.mark.parametrize("n", [1, 2, 31, 33, 1023, 1025, 2047, 2048, 2049, 4095, 4096, 4097,
                               65535, 65536, 65537])
def test_tick_at_size_edges(oracle, n, kind):
    a, b = _particles(n, kind), _particles(n, kind)
    theta = 1.0
    ro = oracle.tick(a, theta=theta)
    with P.Context(n, theta=theta) as ctx:
        codes = np.zeros(n, np.uint32)
        ctx.tick(b, codes)
        t = ctx.tree()
    assert np.array_equal(codes, ro["codes"])
    for k in ("x", "y", "z", "mass", "id"):
        assert np.array_equal(getattr(a, k), getattr(b, k)), k
    for k in TOPO:
        assert np.array_equal(t[k], ro["tree"][k]), k
    assert np.array_equal(t["mp"], ro["tree"]["mp"])
    F = np.stack([b.fx, b.fy, b.fz], 1).astype(np.float64)
    G = np.stack([a.fx, a.fy, a.fz], 1).astype(np.float64)
    assert rel_l2(F, G) < FORCE_REL_L2 or np.abs(G).max() == 0.0


@pytest.mark.parametrize("n", [5, 4096, 32768, 32769])
@pytest.mark.parametrize("mixed", [False, True], ids=["pageable", "one_on_device"])
def test_pageable_arrays_equal_device_arrays(n, mixed):
    torch = pytest.importorskip("torch")

    class D:
        pass

    p, d = _particles(n, "uniform"), D()
    for k in ("x", "y", "z", "mass", "fx", "fy", "fz"):
        setattr(d, k, torch.from_numpy(getattr(p, k).copy()).cuda())
    d.id = torch.from_numpy(p.id.view(np.int32).copy()).cuda()
    if mixed:
        p.fy = torch.zeros(n, device="cuda")
    dc = torch.zeros(n, dtype=torch.int32, device="cuda")
    hc = np.zeros(n, np.uint32)
    torch.cuda.synchronize()
    with P.Context(max(n, 40000), theta=2.0) as ctx:
        for _ in range(2):  # the second on what the first sorted
            ctx.tick(d, dc)
            ctx.tick(p, hc)
    for k in ("x", "y", "z", "mass", "fx", "fy", "fz"):
        h = getattr(p, k)
        h = h.cpu().numpy() if hasattr(h, "cpu") else h
        assert np.array_equal(h, getattr(d, k).cpu().numpy()), k
    assert np.array_equal(p.id, d.id.cpu().numpy().view(np.uint32))
    assert np.array_equal(hc, dc.cpu().numpy().view(np.uint32))
