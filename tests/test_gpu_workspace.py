"""One workspace serves every call that brings data of its own (direct sums, the
closure's features, network, gradient and training): calls of different kinds and
sizes in turn give what a new context gives, and a large one is given back."""

from __future__ import annotations

import numpy as np
import pytest

import polesitter_b200 as P
from conftest import rel_l2
from polesitter_b200 import closure
from polesitter_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _calls(n):
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, 16)).astype(np.float32)
    t = rng.standard_normal((n, 3)).astype(np.float32)
    w = closure.init_params(0)
    p = W.plummer(2048, 51)
    tg = np.arange(min(n, 2048), dtype=np.uint32)
    return {
        "direct": lambda c: c.direct_f64(p, tg),
        "forward": lambda c: c.closure_forward(x, w),
        "grad": lambda c: c.closure_grad(x, t, w)[0],
        "train": lambda c: c.closure_train(x, t, w, 2, 128, 1e-3)[0],
    }


def test_calls_in_turn_equal_new_contexts():
    order = [(300, "train"), (5000, "forward"), (1, "grad"), (700, "direct"), (5000, "grad"),
             (33, "forward"), (2048, "direct"), (1, "train"), (129, "grad"), (1, "direct")]
    p = W.clumpy_plummer(2048, 52)
    with P.Context(2048, theta=4.0) as ctx:
        ctx.set_closure(1)
        ctx.tick(p, np.zeros(p.n, np.uint32))
        idx = np.arange(0, 2048, 7, dtype=np.uint32)
        f0, s0 = ctx.closure_features(idx)
        for n, kind in order:
            got = _calls(n)[kind](ctx)
            if kind == "direct":  # (it takes the context's particle scratch)
                ctx.tick(p, np.zeros(p.n, np.uint32))
            f1, s1 = ctx.closure_features(idx)
            assert np.array_equal(f0, f1) and np.array_equal(s0, s1), (n, kind)
            with P.Context(2048) as fresh:
                want = _calls(n)[kind](fresh)
            if kind in ("direct", "forward"):
                assert np.array_equal(got, want), (n, kind)
            else:  # sums of FP32 atomics, in no fixed order (a few hundred terms each)
                assert rel_l2(got, want) < 1e-4, (n, kind)


def test_large_workspace_is_given_back():
    torch = pytest.importorskip("torch")

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    w = closure.init_params(0)
    small, large = np.zeros((5000, 16), np.float32), np.zeros((1 << 20, 16), np.float32)
    with P.Context(1024) as ctx:
        ctx.closure_forward(small, w)
        held = free()
        for _ in range(3):
            ctx.closure_forward(small, w)
        assert free() == held                  # the small one stays
        ctx.closure_forward(large, w)          # 100 MB
        assert free() >= held
