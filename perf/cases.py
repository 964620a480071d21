"""The work that users of polesitter_b200 have it do, as cases that can be timed.

A case is one call (or a few ticks in one call) through the package's public
entry points:

* ``tick``      ps_prepare_particles + ps_calc_forces (``Context.tick``), the
                reference's call: plain far field (mode 0), order-1 local
                expansion (mode 1) or learned closure (mode 2); any theta and
                leaf capacity; device, pinned or pageable arrays.
* ``loop``      the caller's Euler loop kept on the device
                (``Context.run_ticks``).
* ``ensemble``  many independent systems per tick (``Ensemble.run``).
* ``direct``    the FP64 direct sum a program checks its errors with
                (``Context.direct_f64``).
* ``train``     new closure weights from given samples
                (``Context.closure_train``: network forward, backward, Adam).

Particles are drawn on the GPU from the seed: uniform cubes, Plummer spheres
and the closure's clumpy Plummer family, as ``polesitter_b200.workloads``
describes them.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import polesitter_b200 as P
from polesitter_b200 import closure

DEV = "cuda"
G_DIRECT_PAIRS = 2.5e11   # pairs up to which exact() sums them (a few seconds)


class _Arrays:
    """x, y, z, mass, fx, fy, fz, id views (ps_particle_arrs_t)."""


# ---- the cases ---------------------------------------------------------------

def listed():
    return [
        # the drop-in call of a C program: a small system in its own (pageable)
        # host arrays, the reference's plain settings
        dict(name="cube_1k_host", kind="tick", dist="cube", n=1024, theta=2.0, cap=1, mode=0,
             kahan=False, where="host"),
        # a plain tick of an odd mid-sized system, arrays on the device
        dict(name="plummer_65k", kind="tick", dist="plummer", n=65537, theta=2.0, cap=1, mode=0,
             kahan=False, where="device"),
        # the plain tick at scale: the configuration the parity tests pin
        dict(name="plummer_1m", kind="tick", dist="plummer", n=1 << 20, theta=2.0, cap=1, mode=0,
             kahan=False, where="device"),
        # the plain far field asked for more accuracy: wide theta on the
        # reference's tree, clustered particles, ragged size
        dict(name="clumpy_100k_theta8", kind="tick", dist="clumpy", n=100003, theta=8.0, cap=1,
             mode=0, kahan=False, where="device"),
        # the learned closure on a small system (the smoke check's size)
        dict(name="closure_8k", kind="tick", dist="clumpy", n=8192, theta=6.25, cap=16, mode=2,
             kahan=False, where="device"),
        # ... on an ordinary, ragged one
        dict(name="closure_131k", kind="tick", dist="clumpy", n=131071, theta=6.25, cap=16,
             mode=2, kahan=False, where="device"),
        # ... and the benchmark's headline tick
        dict(name="closure_1m", kind="tick", dist="clumpy", n=1 << 20, theta=6.25, cap=16, mode=2,
             kahan=False, where="device"),
        # the order-1 expansion without the network at the 1e-3 bound, pinned
        # host arrays copied in and out of every tick
        dict(name="order1_250k_pinned", kind="tick", dist="clumpy", n=250000, theta=10.0, cap=16,
             mode=1, kahan=False, where="pinned"),
        # the simulation loop on the device: two colliding Plummer spheres
        dict(name="loop_4m", kind="loop", n=1 << 22, theta=2.0, cap=1, ticks=2),
        # a batch of uneven systems, at the settings its autotuner picks for a
        # 3e-2 error: order-1 expansion, theta 2, leaves of up to 32
        dict(name="ensemble_64", kind="ensemble", systems=64, n_min=1024, n_max=262144, theta=2.0,
             cap=32, order=1, ticks=2),
        # the error check of a 1M tick: FP64 direct sums on 4096 particles
        dict(name="direct_1m", kind="direct", n=1 << 20, targets=4096),
        # new closure weights: two epochs over 128K samples
        dict(name="train_131k", kind="train", n=131072, batch=4096, epochs=2),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(("tick", "loop", "ensemble", "direct", "train"),
                       (0.7, 0.1, 0.1, 0.05, 0.05))[0]
    if kind == "tick":
        mode = rng.choice((0, 0, 0, 1, 2, 2))
        where = rng.choices(("device", "pinned", "host"), (0.6, 0.2, 0.2))[0]
        dist = rng.choice(("cube", "plummer", "clumpy"))
        if mode == 0:
            theta = rng.choice((1.0, 1.5, 2.0, 2.0, 3.0, 4.0, 8.0, 12.0))
            cap = rng.choice((1, 1, 1, 16, 32)) if theta <= 4.0 else 1
            top = 1 << 20 if theta <= 2.0 else 1 << 18 if theta <= 4.0 else 100000
            if theta > 8.0:
                top = 50000
        else:
            theta = rng.choice((5.5, 6.0, 6.25, 6.5, 8.0, 10.0)) if mode == 1 else \
                rng.choice((6.0, 6.25, 6.5))
            cap = rng.choice((8, 16, 16, 24, 32))
            top = 1 << 19 if theta <= 6.5 else 1 << 18 if cap <= 16 else 1 << 17
        return dict(kind="tick", dist=dist, n=_log_int(rng, 1024, top), theta=theta, cap=cap,
                    mode=mode, kahan=mode == 0 and rng.random() < 0.1, where=where)
    if kind == "loop":
        return dict(kind="loop", n=_log_int(rng, 4096, 1 << 21),
                    theta=rng.choice((1.0, 1.5, 2.0)), cap=rng.choice((1, 1, 16)),
                    ticks=rng.randint(1, 4))
    if kind == "ensemble":
        return dict(kind="ensemble", systems=rng.randint(8, 64), n_min=1024,
                    n_max=_log_int(rng, 8192, 262144), theta=rng.choice((1.5, 2.0, 3.0)),
                    cap=rng.choice((1, 16, 32)), order=rng.randint(0, 1),
                    ticks=rng.randint(1, 2))
    if kind == "direct":
        return dict(kind="direct", n=_log_int(rng, 4096, 1 << 20), targets=rng.randint(100, 4096))
    return dict(kind="train", n=_log_int(rng, 8192, 131072), batch=rng.choice((1024, 2048, 4096)),
                epochs=rng.randint(1, 2))


# ---- particles, drawn on the GPU -----------------------------------------------

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _uniform(g, *shape):
    return torch.rand(shape, generator=g, device=DEV, dtype=torch.float64)


def _directions(g, n):
    cz = 2.0 * _uniform(g, n) - 1.0
    phi = 2.0 * math.pi * _uniform(g, n)
    s = torch.sqrt(torch.clamp(1.0 - cz * cz, min=0.0))
    return torch.stack((s * torch.cos(phi), s * torch.sin(phi), cz))


def _plummer(g, n, a=1.0, rmax=10.0):
    """n positions of a Plummer sphere of scale a, radii up to rmax * a."""
    u = _uniform(g, n) * (1.0 + 1.0 / rmax ** 2) ** -1.5
    r = a / torch.sqrt(torch.clamp(u, min=1e-12) ** (-2.0 / 3.0) - 1.0)
    return _directions(g, n) * r


def _clumpy(g, n, clumps=32, fraction=0.3):
    """A Plummer sphere with a fraction of its particles in small clumps."""
    m = int(round(n * fraction))
    centres = _plummer(g, clumps, 1.0, 5.0)
    lo, hi = math.log(0.02), math.log(0.1)
    scales = torch.exp(lo + (hi - lo) * _uniform(g, clumps))
    k = torch.arange(m, device=DEV) % clumps
    return torch.cat((_plummer(g, n - m), _plummer(g, m) * scales[k] + centres[:, k]), 1)


def _positions(g, dist, n):
    if dist == "cube":
        return 2.0 * _uniform(g, 3, n) - 1.0
    return _plummer(g, n) if dist == "plummer" else _clumpy(g, n)


def _speeds(g, n):
    """q = v / v_esc of the isotropic Plummer distribution function, density
    q^2 (1 - q^2)^3.5, by its inverse distribution on a grid."""
    q = torch.linspace(0.0, 1.0, 4097, device=DEV, dtype=torch.float64)
    f = q ** 2 * (1.0 - q ** 2) ** 3.5
    c = torch.cat((torch.zeros(1, device=DEV, dtype=torch.float64),
                   torch.cumsum(0.5 * (f[1:] + f[:-1]), 0)))
    c = c / c[-1]
    u = _uniform(g, n)
    i = torch.clamp(torch.searchsorted(c, u), 1, 4096)
    w = (u - c[i - 1]) / torch.clamp(c[i] - c[i - 1], min=1e-300)
    return q[i - 1] + w * (q[i] - q[i - 1])


def _block(pos, mass):
    """Rows x, y, z, mass, id bits (float32): what a caller hands over."""
    n = pos.shape[1]
    b = torch.empty((5, n), dtype=torch.float32, device=DEV)
    b[:3] = pos
    b[3] = mass
    b[4].view(torch.int32).copy_(torch.arange(n, dtype=torch.int32, device=DEV))
    return b


def _tick_input(case, seed):
    g = _gen(seed)
    pos = _positions(g, case["dist"], case["n"])
    if case["dist"] == "cube":
        return _block(pos, 0.5 + _uniform(g, case["n"]))
    return _block(pos, 1.0 / case["n"])


def _device_arrays(block):
    a = _Arrays()
    a.x, a.y, a.z, a.mass = block[0], block[1], block[2], block[3]
    a.id = block[4].view(torch.int32)
    n = block.shape[1]
    a.fx, a.fy, a.fz = (torch.zeros(n, device=DEV) for _ in range(3))
    return a


def _host_arrays(block, pinned):
    a = _Arrays()
    n = block.shape[1]
    host = block.cpu()

    def array(src=None, dtype=torch.float32):
        t = torch.zeros(n, dtype=dtype, pin_memory=pinned)
        if src is not None:
            t.copy_(src)
        return t.numpy()

    a.x, a.y, a.z, a.mass = (array(host[k]) for k in range(4))
    a.id = array(host[4].view(torch.int32), torch.int32).view(np.uint32)
    a.fx, a.fy, a.fz = (array() for _ in range(3))
    return a, array(dtype=torch.int32).view(np.uint32)


# ---- preparation -----------------------------------------------------------------

def prepare(case, seed):
    return {"tick": _prepare_tick, "loop": _prepare_loop, "ensemble": _prepare_ensemble,
            "direct": _prepare_direct, "train": _prepare_train}[case["kind"]](case, seed)


def _prepare_tick(case, seed):
    block = _tick_input(case, seed)
    n = case["n"]
    ctx = P.Context(n, theta=case["theta"])
    ctx.set_option(P.OPT_LEAF_CAP, case["cap"])
    ctx.set_option(P.OPT_KAHAN, int(case["kahan"]))
    if case["mode"] == 2:
        ctx.closure_set_weights(closure.load(closure.default_weights_path())[0])
    if case["mode"]:
        ctx.set_closure(case["mode"])
    s = dict(kind="tick", ctx=ctx, where=case["where"])
    if case["where"] == "device":
        # the program's own copy of the positions, and the block that the
        # tick sorts in place
        s["fresh"], s["block"] = block, block.clone()
        s["arrays"] = _device_arrays(s["block"])
        s["codes"] = torch.zeros(n, dtype=torch.int32, device=DEV)
    else:
        s["arrays"], s["codes"] = _host_arrays(block, case["where"] == "pinned")
    return s


def _prepare_loop(case, seed):
    g = _gen(seed)
    n = case["n"]
    # two spheres, mass ratio 3:1, 20 apart, closing at 0.3
    n1 = int(round(0.75 * n))
    pos, vel = [], []
    for cnt, mass, x0, v0 in ((n1, 0.75, -5.0, 0.075), (n - n1, 0.25, 15.0, -0.225)):
        p = _plummer(g, cnt)
        v = _directions(g, cnt) * _speeds(g, cnt) * math.sqrt(2.0 * mass) * \
            ((p * p).sum(0) + 1.0) ** -0.25
        p[0] += x0
        v[0] += v0
        pos.append(p)
        vel.append(v)
    ctx = P.Context(n, theta=case["theta"])
    ctx.set_option(P.OPT_LEAF_CAP, case["cap"])
    v = torch.cat(vel, 1).to(torch.float32)
    return dict(kind="loop", ctx=ctx, arrays=_device_arrays(_block(torch.cat(pos, 1), 1.0 / n)),
                codes=torch.zeros(n, dtype=torch.int32, device=DEV), v=[v[c] for c in range(3)],
                ticks=case["ticks"])


def _counts(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    u = rng.uniform(math.log(case["n_min"]), math.log(case["n_max"]), size=case["systems"])
    return np.exp(u).astype(np.int64)


def _prepare_ensemble(case, seed):
    # the batch's sizes belong to the case, its particles to the seed
    counts = _counts(case, case["systems"])
    g = _gen(seed)
    blocks, vel = [], []
    for k, n in enumerate(int(c) for c in counts):
        if k % 2 == 0:  # a uniform cube at rest
            blocks.append(_block(2.0 * _uniform(g, 3, n) - 1.0, (0.5 + _uniform(g, n)) / n))
            vel.append(torch.zeros((3, n), device=DEV))
        else:           # a Plummer sphere of scale 0.5 to 2
            a = 0.5 + 1.5 * (k % 16) / 16.0
            p = _plummer(g, n, a)
            v = _directions(g, n) * _speeds(g, n) * math.sqrt(2.0) * \
                ((p * p).sum(0) + a * a) ** -0.25
            blocks.append(_block(p, 1.0 / n))
            vel.append(v.to(torch.float32))
    block, v = torch.cat(blocks, 1), torch.cat(vel, 1)
    ens = P.Ensemble(counts, np.full(len(counts), case["theta"], np.float32))
    ens.set_order(case["order"])
    ens.set_leaf_caps(np.full(len(counts), case["cap"], np.uint32))
    return dict(kind="ensemble", ens=_Owned(ens), arrays=_device_arrays(block),
                codes=torch.zeros(block.shape[1], dtype=torch.int32, device=DEV),
                v=[v[c] for c in range(3)], ticks=case["ticks"])


class _Owned:
    """An Ensemble that is destroyed with the state that holds it."""

    def __init__(self, ens):
        self.ens = ens

    def __del__(self):
        self.ens.destroy()


def _prepare_direct(case, seed):
    g = _gen(seed)
    n = case["n"]
    arrays = _device_arrays(_block(_clumpy(g, n), 1.0 / n))
    rng = np.random.Generator(np.random.PCG64(seed))
    targets = np.sort(rng.choice(n, size=min(n, case["targets"]), replace=False))
    return dict(kind="direct", ctx=P.Context(n), arrays=arrays, targets=targets.astype(np.uint32))


def _prepare_train(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    n = case["n"]
    # samples of the features' shape: unit-scale field and gradient, offset in
    # the leaf, depth / 10; targets a smooth function of them plus noise
    x = np.zeros((n, 16), np.float32)
    x[:, :9] = 0.3 * rng.standard_normal((n, 9), dtype=np.float32)
    x[:, 9:12] = rng.uniform(-1.0, 1.0, size=(n, 3))
    x[:, 12] = 0.1 * rng.integers(3, 11, size=n)
    t = 2.0 * np.tanh(x[:, 3:6] * x[:, 9:12] * 4.0) + x[:, :3] + \
        0.5 * rng.standard_normal((n, 3), dtype=np.float32)
    return dict(kind="train", ctx=P.Context(1024), x=x, t=np.ascontiguousarray(t, np.float32),
                params=closure.init_params(0), epochs=case["epochs"], batch=case["batch"])


# ---- one pass --------------------------------------------------------------------

def run(state):
    kind = state["kind"]
    if kind == "direct":
        return state["ctx"].direct_f64(state["arrays"], state["targets"])
    if kind == "train":
        params, losses = state["ctx"].closure_train(state["x"], state["t"], state["params"],
                                                    state["epochs"], state["batch"], 2e-3, 0)
        return dict(params=params, losses=losses)
    a, codes = state["arrays"], state["codes"]
    if kind == "tick":
        if state["where"] == "device":
            # a new snapshot arrives in the arrays; the tick runs on its own
            # stream, so the copy has to be over when it is called
            state["block"].copy_(state["fresh"])
            torch.cuda.current_stream().synchronize()
        state["ctx"].tick(a, codes)
    elif kind == "loop":
        state["ctx"].run_ticks(a, codes, *state["v"], 1e-3, state["ticks"])
    else:
        state["ens"].ens.run(a, codes, *state["v"], 1e-3, state["ticks"])
    out = dict(x=a.x, y=a.y, z=a.z, mass=a.mass, id=a.id, codes=codes, fx=a.fx, fy=a.fy, fz=a.fz)
    if kind != "tick":
        out.update(vx=state["v"][0], vy=state["v"][1], vz=state["v"][2])
    elif state["where"] != "device":  # (uint32 bits as int32, as on the device)
        out["id"], out["codes"] = a.id.view(np.int32), codes.view(np.int32)
    return out


# ---- the work a pass cannot do without -----------------------------------------------

def _tick_pairs(n, theta, cap):
    """(M2L pairs, P2P particle pairs) per particle of the method's interaction
    set, as counted on the CPU oracle's trees (n 1024 .. 524,288, theta 1 ..
    10, leaf capacity 1 .. 32; within a factor of two)."""
    t3 = theta ** 3
    nodes = 1.4 if cap == 1 else 3.7 / cap
    p2p = 1.5 * t3 * (1.0 if cap == 1 else 1.2 * cap)
    m2l = 17.0 * t3
    return nodes / 1.4 * m2l / (1.0 + m2l / (nodes * n)), p2p / (1.0 + p2p / n)


def _tick_work(n, theta, cap, order):
    m2l, p2p = _tick_pairs(n, theta, cap)
    # positions, mass, ids in; the same sorted, codes and forces out
    return 56.0 * n, n * ((59.0 if order else 35.0) * m2l + 20.0 * p2p)


def work(case):
    kind = case["kind"]
    if kind == "direct":
        return dict(bytes=16.0 * case["n"] + 28.0 * case["targets"],
                    flops=20.0 * case["n"] * case["targets"])
    if kind == "train":
        steps = case["epochs"] * math.ceil(case["n"] / case["batch"])
        return dict(bytes=case["epochs"] * 80.0 * case["n"] + steps * 28.0 * 9928,
                    flops=case["epochs"] * case["n"] * 6.0 * 9928)
    if kind == "tick":
        b, f = _tick_work(case["n"], case["theta"], case["cap"], case["mode"])
        if case["mode"] == 2:  # the network, and the judge's 1024 direct sums
            f += case["n"] * (2.0 * 9928 + 20.0 * min(1024, case["n"]))
        return dict(bytes=b, flops=f)
    if kind == "loop":
        b, f = _tick_work(case["n"], case["theta"], case["cap"], 0)
        return dict(bytes=case["ticks"] * (b + 24.0 * case["n"]), flops=case["ticks"] * f)
    b = f = 0.0
    for n in _counts(case, case["systems"]):
        bk, fk = _tick_work(float(n), case["theta"], case["cap"], case["order"])
        b, f = b + bk + 24.0 * n, f + fk
    return dict(bytes=case["ticks"] * b, flops=case["ticks"] * f)


# ---- the same in 64 bits ---------------------------------------------------------------

def _morton(pos, n):
    """30-bit codes of the float32 positions, quantised as the x86 reference
    rounds: full groups of 8 to the nearest, the rest truncated."""
    mn, mx = pos.min(), pos.max()
    rng = torch.clamp(mx - mn, min=0.001)
    near = torch.round(torch.clamp((pos - mn) * (1023.0 / rng), 0.0, 1023.0))
    rest = torch.clamp(torch.trunc(((pos - mn) / rng) * 1023.0), 0.0, 1023.0)
    q = torch.where(torch.arange(n, device=pos.device) < n // 8 * 8, near, rest).to(torch.int64)
    code = torch.zeros(n, dtype=torch.int64, device=pos.device)
    for bit in range(10):
        for c in range(3):
            code |= ((q[c] >> bit) & 1) << (3 * bit + c)
    return code


def _direct(pos, mass, targets):
    """FP64 direct-sum forces on the targets (softening 0.1 as float32)."""
    p, m = pos.double(), mass.double()
    eps = float(np.float32(0.1))
    out = torch.empty((3, len(targets)), dtype=torch.float64, device=p.device)
    step = max(1, int(2e8 // p.shape[1]))
    for k in range(0, len(targets), step):
        t = targets[k:k + step]
        d = p[:, None, :] - p[:, t, None]
        w = m / ((d * d).sum(0) + eps) ** 1.5
        out[:, k:k + step] = (d * w).sum(2) * m[t]
    return out


def exact(case, seed):
    n = case["n"] if "n" in case else 0
    if case["kind"] == "direct":
        if n * case["targets"] > G_DIRECT_PAIRS:
            return None
        s = _prepare_direct(case, seed)
        a = s["arrays"]
        t = torch.from_numpy(s["targets"].astype(np.int64)).to(DEV)
        return _direct(torch.stack((a.x, a.y, a.z)), a.mass, t).t().contiguous()
    # the loop's and the ensemble's later orders follow from their own forces,
    # training from its own rounding: no 64-bit value to lay beside them; the
    # forces of the largest ticks would take minutes to sum
    if case["kind"] != "tick" or float(n) * n > G_DIRECT_PAIRS:
        return None
    b = _tick_input(case, seed)
    code = _morton(b[:3], n)
    order = torch.sort(code, stable=True).indices
    b = b[:, order].contiguous()
    f = _direct(b[:3], b[3], torch.arange(n, device=DEV))
    return dict(x=b[0].double(), y=b[1].double(), z=b[2].double(), mass=b[3].double(), id=None,
                codes=None, fx=f[0], fy=f[1], fz=f[2])
