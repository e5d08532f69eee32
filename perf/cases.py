"""What the framework's speed is measured on.

Every case is a whole pass as a user's program makes it, through the Python
solver interface, and can be repeated: it puts a given state in (device arrays
or host arrays), advances it, and takes the result out.  The sizes are those
of the workload configurations (16,000 to 3.35 million particles, batches of
cube scenes, the differentiable 65,536-particle dam break) and sizes between
and below them.

Two kinds of state occur: `fresh`, a lattice block as the scene generators
place it, at rest, jittered by a tenth of its spacing; and `flow`, a
compressed, disordered block in motion, as a scene looks after many sub-steps
(uneven neighbour counts, candidates that differ between neighbouring
particles).
"""
import functools
import math

import numpy as np
import torch

from simplefluid_gb300 import SPHParameters, SPHSolver
from simplefluid_gb300 import _capi as C
from simplefluid_gb300.solver import FRAME_TIME, SPHBatch, batch_cubes

_DT = 1e-4


def listed():
    return [
        # the smallest call: a small drop, one sub-step between two device transfers (latency and launches)
        {"name": "drop_1k_x1", "kind": "step", "layout": "dam", "n": 1331, "state": "fresh", "steps": 1},
        # the 16,000-particle dam break, stepped in a batch of sub-steps as a real-time program does
        {"name": "dambreak_16k_x20", "kind": "step", "layout": "dam", "n": 16000, "state": "fresh", "steps": 20},
        # a 1/30 s frame of the same scene on the device, with the adaptive sub-step: the headless frame loop
        {"name": "frame_16k_adaptive", "kind": "frame", "layout": "dam", "n": 16000, "state": "fresh"},
        # the 65,536-particle dam break in motion, with the Tait equation of state
        {"name": "dambreak_64k_tait_x20", "kind": "step", "layout": "dam", "n": 65536, "state": "flow", "steps": 20,
         "eos": "tait"},
        # an odd size between the named workloads, with attractive pressure
        {"name": "dambreak_237k_flow_x10", "kind": "step", "layout": "dam", "n": 236_987, "state": "flow",
         "steps": 10, "attractive": True},
        # the headline workload at its start: 1,048,576 particles, two dams
        {"name": "double_dam_1m_x10", "kind": "step", "layout": "double", "n": 1_048_576, "state": "fresh",
         "steps": 10},
        # the same size later in a run: disordered and moving
        {"name": "double_dam_1m_flow_x10", "kind": "step", "layout": "double", "n": 1_048_576, "state": "flow",
         "steps": 10},
        # the largest scene: the sphere over the pool
        {"name": "pool_3m_x5", "kind": "step", "layout": "pool", "n": 3_345_599, "state": "fresh", "steps": 5},
        # a program that holds its particles in host memory and reads them back after every sub-step
        {"name": "host_loop_1m_x1", "kind": "host", "layout": "double", "n": 1_048_576, "state": "fresh", "steps": 1},
        # many independent scenes advanced together, host arrays in and out
        {"name": "batch_64_cubes_x40", "kind": "batch", "scenes": 64, "state": "fresh", "steps": 40},
        # one training pass of the differentiable workload: forward with checkpoints, loss, adjoint
        {"name": "adjoint_64k_x40", "kind": "adjoint", "layout": "dam", "n": 65536, "state": "flow", "steps": 40,
         "ckpt": 20},
    ]


def draw(rng):
    """One more case of the same ranges; it costs no more than the largest listed one."""
    def log_int(a, b):
        return max(a, min(b, int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))))

    kind = rng.choice(["step", "step", "step", "step", "frame", "host", "batch", "adjoint"])
    state = rng.choice(["fresh", "flow"])
    if kind == "batch":
        return {"kind": kind, "scenes": log_int(8, 48), "state": state, "steps": log_int(5, 30),
                "scene_seed": rng.randrange(1, 10 ** 6)}
    if kind == "frame":
        return {"kind": kind, "layout": "dam", "n": log_int(1000, 20000), "state": state}
    if kind == "adjoint":
        steps = log_int(10, 40)
        return {"kind": kind, "layout": "dam", "n": log_int(8000, 70000), "state": state, "steps": steps,
                "ckpt": rng.choice([10, 20])}
    n = log_int(1000, 3_345_599)
    layout = rng.choice(["dam", "double"]) if n < 400_000 else rng.choice(["double", "pool"])
    case = {"kind": kind, "layout": layout, "n": n, "state": state,
            "steps": 1 if kind == "host" else log_int(1, max(1, min(20, 16_000_000 // n)))}
    if kind == "step":
        option = rng.choice(["", "", "tait", "attractive", "cells1", "cells3"])
        if option == "tait":
            case["eos"] = "tait"
        elif option == "attractive":
            case["attractive"] = True
        elif option.startswith("cells"):
            case["cells"] = int(option[5:])
    return case


# ---------------------------------------------------------------- scenes
def _radius(case):
    """Particle radius at which the layout holds n particles in the unit box (16,000: 0.01, 65,536 and 1M as the
    named workloads)."""
    n = case["n"]
    if case["layout"] == "pool":
        return ((0.3 + 4.0 / 3.0 * math.pi * 0.15 ** 3) / (8.0 * n)) ** (1.0 / 3.0)
    per = n if case["layout"] == "dam" else (n + 1) // 2
    a = _side(per)
    return (0.4 if case["layout"] == "dam" and n < 40000 else 0.32) / (2.0 * a)


def _side(n):
    a = 1
    while 2 * a ** 3 < n:
        a += 1
    return a


def _params(case):
    r = _radius(case)
    return SPHParameters(
        particleRadius=r, kernelRadius=4.0 * r, pressureStiffness=50.0, viscosity=0.01, restDensity=1000.0,
        timeStep=_DT, boundaryRestitution=0.1,
        eos=C.SF_EOS_TAIT if case.get("eos") == "tait" else C.SF_EOS_LINEAR,
        bUseAttractivePressure=bool(case.get("attractive")), cellsPerH=int(case.get("cells", 2)),
        adaptiveTimeStep=case["kind"] == "frame")


def _block(n, r, corner):
    """First n points (y slowest) of an a x 2a x a lattice at spacing 2r in a corner of the unit box's floor."""
    a = _side(n)
    t = torch.arange(n, device="cuda", dtype=torch.int64)
    x = torch.stack([t % a, t // (a * a), (t // a) % a], 1).double() * (2.0 * r) + r
    if corner:
        x[:, 0] = 1.0 - x[:, 0]
        x[:, 2] = 1.0 - x[:, 2]
    return x


def _pool(n, r):
    s = 2.0 * r
    m, depth = int(1.0 / s), int(math.ceil(0.3 / s))
    t = torch.arange(m * m * depth, device="cuda", dtype=torch.int64)
    pool = torch.stack([t % m, t // (m * m), (t // m) % m], 1).double() * s + r
    k = int(0.34 / s)
    t = torch.arange(k ** 3, device="cuda", dtype=torch.int64)
    ball = (torch.stack([t % k, t // (k * k), (t // k) % k], 1).double() - (k - 1) / 2.0) * s
    ball = ball[ball.square().sum(1) <= 0.155 ** 2] + torch.tensor([0.5, 0.6, 0.5], device="cuda",
                                                                   dtype=torch.float64)
    ball = ball[:n // 2]
    pool = pool[:n - ball.shape[0]]
    if pool.shape[0] + ball.shape[0] < n:  # rounding of the lattice: the rest goes on top of the pool
        rest = n - pool.shape[0] - ball.shape[0]
        t = torch.arange(rest, device="cuda", dtype=torch.int64)
        top = torch.stack([t % m, depth + t // (m * m), (t // m) % m], 1).double() * s + r
        pool = torch.cat([pool, top])
    return torch.cat([pool, ball])


def _disturb(x, r, state, gen, lo, hi):
    """Jitter, and for `flow` compression and motion: float32 (positions, velocities) in the given box."""
    n = x.shape[0]
    amp = (0.1 if state == "fresh" else 0.3) * 2.0 * r
    u = torch.rand((n, 3), generator=gen, device="cuda", dtype=torch.float64) * 2.0 - 1.0
    x = x.clone()
    v = torch.zeros_like(x)
    if state == "flow":
        x[:, 1] = lo + (x[:, 1] - lo) * 0.93
        w = 2.0 * math.pi / (hi - lo)
        v[:, 0] = 0.6 * torch.sin(w * x[:, 1]) * torch.cos(w * x[:, 2])
        v[:, 1] = -0.8 + 0.3 * torch.cos(w * x[:, 0])
        v[:, 2] = 0.4 * torch.sin(w * x[:, 0])
        v += 0.05 * torch.randn((n, 3), generator=gen, device="cuda", dtype=torch.float64)
    x = (x + amp * u).clamp(lo + r, hi - r)
    return x.float().contiguous(), v.float().contiguous()


def _state(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1_000_003 * (int(seed) + 1) + case["n"])
    n, r = case["n"], _radius(case)
    if case["layout"] == "dam":
        x = _block(n, r, False)
    elif case["layout"] == "double":
        x = torch.cat([_block((n + 1) // 2, r, False), _block(n // 2, r, True)])
    else:
        x = _pool(n, r)
    return _disturb(x, r, case["state"], gen, 0.0, 1.0)


_BATCH_BASE = dict(particleRadius=0.005, kernelRadius=0.02, pressureStiffness=50.0, viscosity=0.01,
                   restDensity=1000.0, timeStep=_DT, boundaryRestitution=0.1)


@functools.lru_cache(maxsize=4)
def _cubes(scene_seed, scenes):
    params, counts, pos = batch_cubes(scene_seed, scenes, SPHParameters(**_BATCH_BASE))
    return [SPHParameters.from_c(p) for p in params], counts, pos


def _batch_state(case, seed):
    params, counts, pos = _cubes(case.get("scene_seed", 20171), case["scenes"])
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1_000_003 * (int(seed) + 1) + case["scenes"])
    xs, vs, at = [], [], 0
    for p, n in zip(params, counts.tolist()):
        x = torch.from_numpy(pos[at:at + n]).cuda().double()
        x, v = _disturb(x, p.particleRadius, case["state"], gen, 0.0, p.boxMax[0])
        xs.append(x)
        vs.append(v)
        at += n
    return params, counts, torch.cat(xs).cpu().numpy(), torch.cat(vs).cpu().numpy()


_HIST = 32  # histogram resolution of the differentiable workload


def _target(seed):
    t = np.random.RandomState(int(seed) % (1 << 31)).random_sample(_HIST ** 3).astype(np.float32)
    return t / t.sum()


# ---------------------------------------------------------------- a pass
def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        params, counts, pos, vel = _batch_state(case, seed)
        return {"case": case, "batch": SPHBatch(params), "counts": counts, "pos": pos, "vel": vel}
    pos, vel = _state(case, seed)
    st = {"case": case, "solver": SPHSolver(_params(case))}
    if kind == "host":
        st["pos"], st["vel"] = pos.cpu().numpy(), vel.cpu().numpy()
        return st
    st["pos"], st["vel"] = pos, vel
    if kind == "adjoint":
        st["target"] = _target(seed)
    else:
        st["out_pos"], st["out_vel"] = torch.empty_like(pos), torch.empty_like(vel)
    return st


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batch":
        b = state["batch"]
        b.setState(state["counts"], state["pos"], state["vel"])
        b.step(case["steps"])
        pos, vel = b.getState()
        return {"pos": pos, "vel": vel}
    s = state["solver"]
    if kind == "host":
        s.setParticles(state["pos"], state["vel"])
        for _ in range(case["steps"]):
            s.advanceFrame()
        pos, vel = s.getState()
        return {"pos": pos, "vel": vel}
    stream = torch.cuda.current_stream()
    s.setParticlesDevice(state["pos"], state["vel"], stream=stream)
    if kind == "adjoint":
        s.forward(case["steps"], case["ckpt"])
        loss, gx = s.lossHistogram(state["target"])
        dx0, dv0, dmu, dk = s.adjoint(gx)
        return {"loss": loss, "dloss_dx": gx, "dx0": dx0, "dv0": dv0, "dviscosity": dmu, "dstiffness": dk}
    out = {"pos": state["out_pos"], "vel": state["out_vel"]}
    if kind == "frame":
        out["time"], out["substeps"] = s.advanceFrames(1, FRAME_TIME)
    else:
        s.step(case["steps"])
    s.getStateDevice(out["pos"], out["vel"], stream=stream)
    return out


# A neighbour's terms: density 12 operations (difference, square, weight, sum), force 34 (the same distance, root,
# quotient, weights, six sums); a particle has about 34 neighbours at spacing 2r and kernel radius 4r.
_PER_UPDATE = 34 * (12 + 34) + 40
_PER_ADJOINT = 34 * (90 + 12) + 100  # the reverse passes of one update


def work(case):
    """One pass: the state in and out once, and the pair terms of every update."""
    if case["kind"] == "batch":
        n, steps = int(_cubes(case.get("scene_seed", 20171), case["scenes"])[1].sum()), case["steps"]
    else:
        n, steps = case["n"], case.get("steps") or int(math.ceil(FRAME_TIME / _DT))
    if case["kind"] == "adjoint":
        # state in; gradients of the last positions, the first positions and velocities out; the target histogram
        return {"bytes": 24 * n + 36 * n + 4 * _HIST ** 3, "flops": n * steps * (2 * _PER_UPDATE + _PER_ADJOINT)}
    return {"bytes": 48 * n, "flops": n * steps * _PER_UPDATE}


# ---------------------------------------------------------------- the same in 64 bits
def _f(v):
    return float(np.float32(v))


def _pairs(x, h):
    """Chunks (i, j) of all pairs closer than h, each particle with itself included."""
    x = x.detach()
    c = ((x - x.min(0).values) / h).floor().long() + 1
    d = c.max(0).values + 2
    key = (c[:, 2] * d[1] + c[:, 1]) * d[0] + c[:, 0]
    ks, order = torch.sort(key)
    out = []
    for at in range(0, x.shape[0], 1 << 17):
        ii = torch.arange(at, min(at + (1 << 17), x.shape[0]), device=x.device)
        gi, gj = [], []
        for dz in (-1, 0, 1):
            for dy in (-1, 0, 1):
                k0 = key[ii] + (dz * d[1] + dy) * d[0] - 1
                b, e = torch.searchsorted(ks, k0), torch.searchsorted(ks, k0 + 3)
                m = e - b
                i = torch.repeat_interleave(ii, m)
                first = torch.repeat_interleave(b - (m.cumsum(0) - m), m)
                j = order[first + torch.arange(i.shape[0], device=x.device)]
                near = (x[i] - x[j]).square().sum(1) < h * h
                gi.append(i[near])
                gj.append(j[near])
        out.append((torch.cat(gi), torch.cat(gj)))
    return out


def _advance(p, x, v, dt, k, mu):
    """One sub-step in 64 bits: (x, v, acceleration).  k and mu may be tensors (for their gradients)."""
    h, r, rho0 = _f(p.kernelRadius), _f(p.particleRadius), _f(p.restDensity)
    mass = rho0 * (2.0 * r) ** 3
    g = torch.tensor([_f(a) for a in p.gravity], device=x.device, dtype=torch.float64)
    chunks = _pairs(x, h)
    s = torch.zeros_like(x[:, 0])
    for i, j in chunks:
        s = s.index_add(0, i, (h * h - (x[i] - x[j]).square().sum(1)) ** 3)
    rho = s * (mass * 315.0 / (64.0 * math.pi * h ** 9))
    prs = k * ((rho / rho0) ** 7 - 1.0) if p.eos == C.SF_EOS_TAIT else k * (rho - rho0)
    if not p.bUseAttractivePressure:
        prs = torch.relu(prs)
    inv = 1.0 / rho
    ap, av = torch.zeros_like(x), torch.zeros_like(x)
    for i, j in chunks:
        far = (i != j) & ((x.detach()[i] - x.detach()[j]).square().sum(1) > 0)
        i, j = i[far], j[far]
        d = x[i] - x[j]
        dist = d.square().sum(1).sqrt()
        w = (h - dist) * inv[j]
        ap = ap.index_add(0, i, ((prs[i] + prs[j]) * w * (h - dist) / dist)[:, None] * d)
        av = av.index_add(0, i, w[:, None] * (v[j] - v[i]))
    cp, cv = mass * 45.0 / (math.pi * h ** 6), mass * 45.0 / (math.pi * h ** 6)
    a = (0.5 * cp * ap + mu * cv * av) * inv[:, None] + g
    v = v + dt * a
    x = x + dt * v
    e = _f(p.boundaryRestitution)
    lo = torch.tensor([_f(b) + r for b in p.boxMin], device=x.device, dtype=torch.float64)
    hi = torch.tensor([_f(b) - r for b in p.boxMax], device=x.device, dtype=torch.float64)
    below, above = x < lo, x > hi
    v = torch.where((below & (v < 0)) | (above & (v > 0)), -e * v, v)
    x = torch.where(below, lo.expand_as(x), torch.where(above, hi.expand_as(x), x))
    return x, v, a


def _steps(p, pos, vel, steps):
    x, v = pos.double(), vel.double()
    with torch.no_grad():
        for _ in range(steps):
            x, v, _a = _advance(p, x, v, _f(p.timeStep), _f(p.pressureStiffness), _f(p.viscosity))
    return x, v


def _frame(p, pos, vel):
    """The frame loop with the adaptive sub-step; the clock adds 32-bit sub-steps, as the frame loop does."""
    x, v = pos.double(), vel.double()
    h, a2, acc, taken = _f(p.kernelRadius), 0.0, np.float32(0.0), 0
    with torch.no_grad():
        while float(acc) < FRAME_TIME:
            v2 = float(v.square().sum(1).max())
            dt = _f(p.timeStep)
            if v2 > 0:
                dt = min(dt, 0.4 * h / math.sqrt(v2))
            if a2 > 0:
                dt = min(dt, 0.25 * math.sqrt(h / math.sqrt(a2)))
            x, v, a = _advance(p, x, v, dt, _f(p.pressureStiffness), _f(p.viscosity))
            a2 = float(a.square().sum(1).max())
            acc = np.float32(acc + np.float32(dt))
            taken += 1
    return x, v, float(acc)


def _histogram_loss(x, target):
    """Squared distance of the cloud-in-cell histogram over the unit box (cell-centred bins) to the target."""
    u = x * _HIST - 0.5
    base = u.detach().floor()
    f = u - base
    hist = torch.zeros(_HIST ** 3, device=x.device, dtype=torch.float64)
    for q in range(8):
        o = torch.tensor([q & 1, (q >> 1) & 1, (q >> 2) & 1], device=x.device)
        c = base.long() + o
        inside = ((c >= 0) & (c < _HIST)).all(1)
        w = torch.where(o.bool(), f, 1.0 - f).prod(1)
        flat = (c[:, 2] * _HIST + c[:, 1]) * _HIST + c[:, 0]
        hist = hist.index_add(0, flat[inside], w[inside])
    return (hist / x.shape[0] - torch.from_numpy(target).to(x.device).double()).square().sum()


def _adjoint(p, pos, vel, steps, target):
    x0, v0 = pos.double().requires_grad_(), vel.double().requires_grad_()
    k = torch.tensor(_f(p.pressureStiffness), device="cuda", dtype=torch.float64, requires_grad=True)
    mu = torch.tensor(_f(p.viscosity), device="cuda", dtype=torch.float64, requires_grad=True)

    def one(x, v, k, mu):
        return _advance(p, x, v, _f(p.timeStep), k, mu)[:2]

    from torch.utils.checkpoint import checkpoint
    x, v = x0, v0
    for _ in range(steps):
        x, v = checkpoint(one, x, v, k, mu, use_reentrant=False)
    loss = _histogram_loss(x, target)
    gx, dx0, dv0, dk, dmu = torch.autograd.grad(loss, [x, x0, v0, k, mu])
    return {"loss": float(loss), "dloss_dx": gx, "dx0": dx0, "dv0": dv0, "dviscosity": float(dmu),
            "dstiffness": float(dk)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        params, counts, pos, vel = _batch_state(case, seed)
        xs, vs, at = [], [], 0
        for p, n in zip(params, counts.tolist()):
            x, v = _steps(p, torch.from_numpy(pos[at:at + n]).cuda(), torch.from_numpy(vel[at:at + n]).cuda(),
                          case["steps"])
            xs.append(x)
            vs.append(v)
            at += n
        return {"pos": torch.cat(xs), "vel": torch.cat(vs)}
    p = _params(case)
    pos, vel = _state(case, seed)
    if kind == "adjoint":
        return _adjoint(p, pos, vel, case["steps"], _target(seed))
    if kind == "frame":
        x, v, t = _frame(p, pos, vel)
        return {"pos": x, "vel": v, "time": t, "substeps": None}
    x, v = _steps(p, pos, vel, case["steps"])
    return {"pos": x, "vel": v}
