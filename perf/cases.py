"""What a user of this engine has it do, as measurable cases through its public entry points.

Every case takes two-disk encounters (exponential disks, circular speeds, the second disk
offset, approaching and inclined -- the systems of this repository's benchmark and tests) made
on the GPU from the seed, and one entry point:

  accel        adjoint.accelerations: one direct sum on CUDA tensors, in FP64, mixed or the
               reference-order ("f64-exact") form
  run          Session.step and Session.diagnostics: the reference program's loop between two
               outputs, state resident on the device
  fmm          fmm.fmm_accelerations: one FMM evaluation on CUDA tensors, statistics included
  fmmrun       Session.set_fmm and Session.step: FMM steps of a resident session
  ensemble     Batch.step: steps of many independent encounters of uneven size
  fit          adjoint.leapfrog and its gradient: one iteration of an orbit fit
  diagnostics  Session.diagnostics: the row of diagnostics.csv

``listed`` gives the named cases, ``draw`` more of the same ranges, ``work`` the bytes and
operations that a pass cannot do without, ``exact`` the values in plain 64-bit torch.
"""
from __future__ import annotations

import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

PAIR_FLOPS = 20      # one softened pair: 3 sub, |d|^2 + eps^2, rsqrt, cube, mass, 3 FMA
POTENTIAL_FLOPS = 11  # one pair of the potential energy
FAR_FLOPS = 250      # one body against one far node at expansion order 4
VJP_FLOPS = 55       # one pair of the adjoint sum
STATE = ("x", "y", "z", "vx", "vy", "vz", "ax", "ay", "az")


def _gx():
    """The package (its folder's name is no identifier), loaded once as ``gx``."""
    if "gx" not in sys.modules:
        root = Path.cwd() / "galaxy-collision-simulation_b200"
        spec = importlib.util.spec_from_file_location("gx", root / "__init__.py",
                                                      submodule_search_locations=[str(root)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["gx"] = mod
        spec.loader.exec_module(mod)
    import gx.adjoint  # noqa: F401  (needs torch, so the package does not import it itself)
    return sys.modules["gx"]


def listed():
    return [
        # the reference's published N = 1000 benchmark: 20 FP64 steps between two outputs, then
        # the diagnostics row; every step is a few microseconds, so launches and waits count
        {"name": "run-f64-n1000", "kind": "run", "n": 1000, "precision": "f64", "steps": 20, "dt": 0.005, "eps": 0.05},
        # the drop-in for compute_cuda_direct_accelerations at an ordinary, ragged size
        {"name": "accel-f64-n49999", "kind": "accel", "n": 49999, "precision": "f64", "eps": 0.02},
        # the same call in mixed precision at the size of the repository's 65,536-body workload
        {"name": "accel-mixed-n65536", "kind": "accel", "n": 65536, "precision": "mixed", "eps": 0.02},
        # the headline workload: one mixed-precision step of 2^20 bodies
        {"name": "run-mixed-n1048576", "kind": "run", "n": 1048576, "precision": "mixed", "steps": 1, "dt": 0.001,
         "eps": 0.01, "rows": False},
        # the parity form (bit-identical to the reference's sum), as a validation run uses it
        {"name": "accel-exact-n16384", "kind": "accel", "n": 16384, "precision": "f64-exact", "eps": 0.02},
        # the reference's 1000-body FMM run with its default options: latency, launches, host reads
        {"name": "fmm-f64-n1000-leaf16", "kind": "fmm", "n": 1000, "precision": "f64", "leaf": 16, "theta": 0.6,
         "order": 4, "eps": 0.05},
        # the 65,536-body FMM workload, one evaluation on the caller's arrays
        {"name": "fmm-f64-n65536-leaf64", "kind": "fmm", "n": 65536, "precision": "f64", "leaf": 64, "theta": 0.6,
         "order": 4, "eps": 0.02},
        # the largest FMM: 2^20 bodies, the reference's default leaf capacity, mixed precision
        {"name": "fmm-mixed-n1048576-leaf16", "kind": "fmm", "n": 1048576, "precision": "mixed", "leaf": 16,
         "theta": 0.6, "order": 4, "eps": 0.01},
        # the same workload as a resident FMM session, where nothing is read back between steps
        {"name": "fmmrun-f64-n65536-leaf64", "kind": "fmmrun", "n": 65536, "precision": "f64", "leaf": 64,
         "theta": 0.6, "order": 4, "steps": 4, "dt": 0.002, "eps": 0.02},
        # a parameter study: 128 encounters of 1024 to 16384 bodies stepped together
        {"name": "ensemble-mixed-128", "kind": "ensemble", "instances": 128, "n_min": 1024, "n_max": 16384,
         "sizes": 11, "precision": "mixed", "steps": 2, "dt": 0.005, "eps": 0.05},
        # one gradient of an orbit fit: forward and backward through checkpointed steps, with
        # FP32 parameters, as mixed-precision fits hold them
        {"name": "fit-mixed-n16384", "kind": "fit", "n": 16384, "precision": "mixed", "steps": 10, "every": 5,
         "dt": 0.005, "eps": 0.05},
        # the diagnostics row of a 65,536-body system, taken with every snapshot
        {"name": "diagnostics-n65536", "kind": "diagnostics", "n": 65536, "eps": 0.02},
    ]


def _size(rng, lo, hi):
    """A size spread over its logarithm; any integer, odd ones included."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "accel", "accel", "fmm", "fmm", "fmmrun", "ensemble", "fit", "diagnostics"])
    c = {"kind": kind}
    if kind == "run":
        c.update(n=_size(rng, 250, 30000), precision=rng.choice(["f64", "mixed", "f64-exact"]),
                 steps=rng.randint(5, 20), dt=0.005, eps=0.05)
    elif kind == "accel":
        p = rng.choice(["f64", "mixed", "f64-exact"])
        c.update(n=_size(rng, 250, 30000 if p == "f64-exact" else 130000), precision=p, eps=0.02)
    elif kind == "fmm":
        c.update(n=_size(rng, 500, 1000000), precision=rng.choice(["f64", "mixed"]), leaf=rng.choice([16, 32, 64]),
                 theta=rng.choice([0.5, 0.6, 0.7]), order=rng.choice([2, 4, 4]), eps=0.02)
    elif kind == "fmmrun":
        c.update(n=_size(rng, 1000, 200000), precision=rng.choice(["f64", "mixed"]), leaf=rng.choice([16, 64]),
                 theta=0.6, order=4, steps=rng.randint(2, 5), dt=0.002, eps=0.02)
    elif kind == "ensemble":
        c.update(instances=rng.randint(8, 128), n_min=1024, n_max=16384, sizes=rng.randrange(1 << 20),
                 precision=rng.choice(["f64", "mixed", "mixed"]), steps=2, dt=0.005, eps=0.05)
    elif kind == "fit":
        c.update(n=_size(rng, 500, 16384), precision=rng.choice(["f64", "mixed"]), steps=rng.randint(4, 10), every=5,
                 dt=0.005, eps=0.05)
    else:
        c.update(n=_size(rng, 250, 130000), eps=0.02)
    return c


# ---- inputs ---------------------------------------------------------------------------------
def _disk(n, mass, g, eps):
    """One face-on exponential disk (scale 1, truncated at 5): positions (3, n), velocities, masses."""
    f = dict(dtype=torch.float64, device="cuda")
    u = torch.rand(n, generator=g, **f)
    target = u * (1.0 - 6.0 * math.exp(-5.0))
    lo, hi = torch.zeros(n, **f), torch.full((n,), 5.0, **f)
    for _ in range(54):
        mid = 0.5 * (lo + hi)
        below = 1.0 - (1.0 + mid) * torch.exp(-mid) < target
        lo, hi = torch.where(below, mid, lo), torch.where(below, hi, mid)
    r = 0.5 * (lo + hi)
    th = 2.0 * math.pi * torch.rand(n, generator=g, **f)
    z = 0.05 * torch.randn(n, generator=g, **f)
    rank = torch.empty(n, **f)
    rank[torch.argsort(r)] = torch.arange(1, n + 1, **f)
    vc = torch.sqrt(rank * (mass / n) * r * r / (r * r + eps * eps) ** 1.5)
    pos = torch.stack([r * torch.cos(th), r * torch.sin(th), z])
    vel = torch.stack([-torch.sin(th) * vc, torch.cos(th) * vc, torch.zeros_like(r)])
    return pos, vel, torch.full((n,), mass / n, **f)


def _encounter(n, seed, eps, mass2=1.0, impact=2.0, inclination=30.0):
    """Two disks: the second at (10, impact, 0), approaching at 0.5 and inclined about x."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    n1 = n - n // 2
    p1, v1, m1 = _disk(n1, 1.0, g, eps)
    p2, v2, m2 = _disk(n // 2, mass2, g, eps)
    a = math.radians(inclination)
    rot = torch.tensor([[1.0, 0.0, 0.0], [0.0, math.cos(a), -math.sin(a)], [0.0, math.sin(a), math.cos(a)]],
                       dtype=torch.float64, device="cuda")
    p2 = rot @ p2 + torch.tensor([[10.0], [impact], [0.0]], dtype=torch.float64, device="cuda")
    v2 = rot @ v2 + torch.tensor([[-0.5], [0.0], [0.0]], dtype=torch.float64, device="cuda")
    return torch.cat([p1, p2], 1).contiguous(), torch.cat([v1, v2], 1).contiguous(), torch.cat([m1, m2])


def _mass2(case):
    return 1.0 / 3.0 if case["n"] > 500000 else 1.0


def _ensemble(case, seed):
    """Offsets (the sizes are the case's own) and the concatenated state: mass ratios, impacts and
    inclinations drawn from the seed."""
    k = case["instances"]
    sizes = 2 * np.random.default_rng(case["sizes"]).integers(case["n_min"] // 2, case["n_max"] // 2 + 1, k)
    rng = np.random.default_rng(seed)
    offsets = np.zeros(k + 1, np.int64)
    offsets[1:] = np.cumsum(sizes)
    parts = [_encounter(int(sizes[b]), int(rng.integers(0, 2**31)), case["eps"], 1.0 / rng.uniform(1.0, 10.0),
                        rng.uniform(0.5, 4.0), rng.uniform(0.0, 90.0)) for b in range(k)]
    return offsets, *(torch.cat([p[c] for p in parts], -1).contiguous() for c in range(3))


class _Resident:
    """A resident array of a session or a batch, for torch.as_tensor (whose tensor keeps this
    object, and with it the owner of the memory, alive)."""

    def __init__(self, owner, address, n):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (address, False), "version": 3}


def _views(owner, n):
    arrays = owner.device_arrays()
    return {k: torch.as_tensor(_Resident(owner, arrays[k], n), device="cuda") for k in STATE}


def _fit_inputs(case, seed):
    """Initial state (n, 3) and masses as parameters of the fit, and the target positions."""
    X, V, m = _encounter(case["n"], seed, case["eps"])
    dtype = torch.float32 if case["precision"] == "mixed" else torch.float64
    x0, v0, m = (t.to(dtype) for t in (X.t().contiguous(), V.t().contiguous(), m))
    target = x0.double() + case["steps"] * case["dt"] * v0.double()
    target[case["n"] // 2:, 1] += 0.1  # the observed encounter has another impact parameter
    return x0, v0, m, target


def prepare(case, seed):
    gx = _gx()
    kind = case["kind"]
    params = gx.PhysicsParams(1.0, case["eps"])
    if kind == "ensemble":
        offsets, X, V, m = _ensemble(case, seed)
        b = gx.Batch(offsets, params)
        torch.cuda.synchronize()  # the batch copies on a stream of its own
        b.set_state(X[0], X[1], X[2], V[0], V[1], V[2], m)
        b.compute_accelerations(case["precision"])
        b.synchronize()
        return {"case": case, "batch": b, "views": _views(b, X.shape[1])}
    if kind == "fit":
        x0, v0, m, target = _fit_inputs(case, seed)
        leaves = [t.requires_grad_(True) for t in (x0, v0, m)]
        return {"case": case, "params": params, "leaves": leaves, "target": target}
    X, V, m = _encounter(case["n"], seed, case["eps"], _mass2(case))
    if kind == "accel":
        return {"case": case, "params": params, "X": X, "m": m}
    if kind == "fmm":
        return {"case": case, "params": params, "X": X, "m": m, "A": torch.zeros_like(X), "opt": _options(gx, case)}
    s = gx.Session(case["n"], params)
    torch.cuda.synchronize()  # the session copies on a stream of its own
    s.set_state(X[0], X[1], X[2], V[0], V[1], V[2], m)
    if kind == "fmmrun":
        s.set_fmm(_options(gx, case))
    if kind != "diagnostics":
        s.compute_accelerations(case["precision"])
    s.synchronize()
    return {"case": case, "session": s, "views": _views(s, case["n"])}


def _options(gx, case):
    return gx.FmmOptions(theta=case["theta"], leaf_capacity=case["leaf"], expansion_order=case["order"])


# ---- one pass -------------------------------------------------------------------------------
def run(state):
    case, gx = state["case"], _gx()
    kind = case["kind"]
    if kind == "accel":
        return gx.adjoint.accelerations(state["X"], state["m"], state["params"], case["precision"])
    if kind == "fmm":
        X, A = state["X"], state["A"]
        st = gx.fmm.fmm_accelerations(X[0], X[1], X[2], state["m"], A[0], A[1], A[2], state["params"], state["opt"],
                                      case["precision"])
        return {"a": A, "stats": [st.node_count, st.leaf_count, st.far_interactions, st.near_interactions,
                                  st.far_pairs, st.near_pairs, st.tree_levels]}
    if kind == "ensemble":
        state["batch"].step(case["steps"], case["dt"], case["precision"])
        return dict(state["views"])
    if kind == "fit":
        x0, v0, m = state["leaves"]
        xT, vT = gx.adjoint.leapfrog(x0, v0, m, case["steps"], case["dt"], state["params"], case["every"],
                                     case["precision"])
        loss = ((xT - state["target"]) ** 2).sum(1).mean()
        gx0, gv0, gm = torch.autograd.grad(loss, (x0, v0, m))
        return {"x": xT.detach(), "v": vT.detach(), "gx": gx0, "gv": gv0, "gm": gm}
    if kind == "diagnostics":
        return np.array(state["session"].diagnostics().as_row())
    s = state["session"]  # the updated state stays in its buffers
    s.step(case["steps"], case["dt"], case["precision"])
    if kind == "run" and case.get("rows", True):
        return {**state["views"], "row": np.array(s.diagnostics().as_row())}
    return dict(state["views"])


# ---- what a pass cannot do without ------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "ensemble":  # sizes are uniform on [n_min, n_max]
        a, b, k, s = case["n_min"], case["n_max"], case["instances"], case["steps"]
        return {"bytes": 152.0 * k * s * (a + b) / 2, "flops": float(PAIR_FLOPS) * k * s * (a * a + a * b + b * b) / 3}
    n = case["n"]
    pairs = float(n) * (n - 1)
    if kind == "accel":
        return {"bytes": 56.0 * n, "flops": PAIR_FLOPS * pairs}
    if kind == "run":
        rows = case.get("rows", True)
        return {"bytes": 152.0 * n * case["steps"] + (56.0 * n if rows else 0.0),
                "flops": PAIR_FLOPS * pairs * case["steps"] + (POTENTIAL_FLOPS * pairs / 2 if rows else 0.0)}
    if kind == "diagnostics":
        return {"bytes": 56.0 * n, "flops": POTENTIAL_FLOPS * pairs / 2}
    if kind == "fit":
        # every state's force forward, again from the checkpoints, and one adjoint sum per state
        s = case["steps"]
        return {"bytes": 152.0 * n * 2 * s + 88.0 * n * (s + 1),
                "flops": pairs * (PAIR_FLOPS * (2 * s + 1) + VJP_FLOPS * (s + 1))}
    # FMM: about 50 leaf capacities of near bodies and 100 far nodes per level and body
    steps = case.get("steps", 1)
    near = min(n, 50.0 * case["leaf"])
    far = 100.0 * max(0.0, math.log(n / case["leaf"], 8)) if n > case["leaf"] else 0.0
    return {"bytes": (56.0 if kind == "fmm" else 152.0) * n * steps,
            "flops": n * steps * (PAIR_FLOPS * near + (FAR_FLOPS if case["order"] == 4 else 80) * far)}


# ---- 64-bit values ----------------------------------------------------------------------------
def _rows_per_chunk(n):
    return max(1, min(n, (1 << 26) // n))


def _accel64(X, m, eps):
    """Direct sum in 64 bits, a block of targets at a time: X (3, n) -> (3, n)."""
    n = X.shape[1]
    out = torch.empty_like(X)
    step = _rows_per_chunk(n)
    for b in range(0, n, step):
        d = X[:, None, :] - X[:, b:b + step, None]
        s = (d * d).sum(0) + eps * eps
        w = m / (s * torch.sqrt(s))
        out[:, b:b + step] = (d * w).sum(2)
    return out


def _vjp64(X, m, lam, eps):
    """Gradients of sum(lam . accelerations) with respect to X and m, in 64 bits."""
    n = X.shape[1]
    gx, gm = torch.empty_like(X), torch.empty_like(m)
    step = max(1, _rows_per_chunk(n) // 2)
    for b in range(0, n, step):
        e = slice(b, b + step)
        d = X[:, None, :] - X[:, e, None]
        s = (d * d).sum(0) + eps * eps
        i3 = 1.0 / (s * torch.sqrt(s))
        A = m[None, e, None] * lam[:, None, :] - m * lam[:, e, None]
        c = 3.0 * (i3 / s) * (A * d).sum(0)
        gx[:, e] = (A * i3 - d * c).sum(2)
        gm[e] = -(i3 * (d * lam[:, None, :]).sum(0)).sum(1)
    return gx, gm


def _row64(X, V, m, eps):
    """The diagnostics row: mass, energies, momentum, centre of mass, angular momentum."""
    n = X.shape[1]
    ke = 0.5 * (m * (V * V).sum(0)).sum()
    pe = torch.zeros((), dtype=torch.float64, device=X.device)
    step = _rows_per_chunk(n)
    for b in range(0, n, step):
        d = X[:, None, :] - X[:, b:b + step, None]
        w = m / torch.sqrt((d * d).sum(0) + eps * eps)
        k = torch.arange(w.shape[0], device=X.device)
        w[k, b + k] = 0.0
        pe -= 0.5 * (m[b:b + step] * w.sum(1)).sum()
    M = m.sum()
    spin = torch.linalg.cross(X.t(), V.t()).t()
    vals = [M, ke, pe, ke + pe, *(V * m).sum(1), *((X * m).sum(1) / M), *(spin * m).sum(1)]
    return torch.stack(vals).cpu().numpy()


def _steps64(X, V, A, m, steps, dt, eps):
    for _ in range(steps):
        V = V + 0.5 * dt * A
        X = X + dt * V
        A = _accel64(X, m, eps)
        V = V + 0.5 * dt * A
    return X, V, A


def _named(X, V, A):
    return {k: t.contiguous() for k, t in zip(STATE, (*X, *V, *A))}


def exact(case, seed):
    kind, eps = case["kind"], case["eps"]
    if kind == "ensemble":
        if case["instances"] > 128:
            return None
        offsets, X, V, m = _ensemble(case, seed)
        A = torch.empty_like(X)
        for b in range(len(offsets) - 1):
            e = slice(int(offsets[b]), int(offsets[b + 1]))
            x, v, mm = X[:, e].contiguous(), V[:, e], m[e]
            X[:, e], V[:, e], A[:, e] = _steps64(x, v, _accel64(x, mm, eps), mm, case["steps"], case["dt"], eps)
        return _named(X, V, A)
    if kind == "fit":
        x0, v0, m, target = _fit_inputs(case, seed)
        n, steps, dt, h = case["n"], case["steps"], case["dt"], 0.5 * case["dt"]
        X, V, m = x0.double().t().contiguous(), v0.double().t().contiguous(), m.double()
        states, A = [X], _accel64(X, m, eps)
        for _ in range(steps):
            X, V, A = _steps64(X, V, A, m, 1, dt, eps)
            states.append(X)
        # the adjoint of kick-drift-kick, last state first (its closing kick has no cotangent: the
        # loss reads positions only)
        xb, vb, mb = (2.0 / n) * (X - target.t()), torch.zeros_like(X), torch.zeros_like(m)
        for k in range(steps - 1, -1, -1):
            vb = vb + dt * xb
            g, gm = _vjp64(states[k], m, (dt if k >= 1 else h) * vb, eps)
            xb, mb = xb + g, mb + gm
        rows = {"x": X, "v": V, "gx": xb, "gv": vb}
        return {**{k: t.t().contiguous() for k, t in rows.items()}, "gm": mb}
    n = case["n"]
    if float(n) * n * case.get("steps", 1) > 5e10:  # beyond about 20 seconds
        return None
    X, V, m = _encounter(n, seed, eps, _mass2(case))
    if kind == "accel":
        return _accel64(X, m, eps)
    if kind == "fmm":  # the sum that the expansion approximates
        return {"a": _accel64(X, m, eps), "stats": None}
    if kind == "diagnostics":
        return _row64(X, V, m, eps)
    X, V, A = _steps64(X, V, _accel64(X, m, eps), m, case["steps"], case["dt"], eps)
    out = _named(X, V, A)
    if kind == "run" and case.get("rows", True):
        out["row"] = _row64(X, V, m, eps)
    return out
