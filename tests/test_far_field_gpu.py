"""Far field over staged node records against Taylor expansions of every far body (B200).

Leaves of 1 to more than a block of targets (a thread block holds 128 / targets node slots, at most
64, and its warps copy node records in passes of a power of two), expansion orders 0, 2 and 4, FP64
and mixed.  A multipole of order p about a centre is, body by body, the order-p Taylor polynomial of
the softened force in the body's offset from the centre; the near field is summed directly.
FP64: 1e-11 of the sum of magnitudes.  Mixed (FP32 terms, about 250 operations each): 1e-5 of it.
"""
import numpy as np
import pytest

import gx

pytestmark = pytest.mark.gpu

EPS, THETA = 0.02, 0.6


def octree(X, m, cap):
    """(beg, end, centre, half width, children) per node and the body order."""
    lo, hi = X.min(0), X.max(0)
    perm, nodes = [], []

    def build(idx, c, hw):
        k = len(nodes)
        node = dict(idx=idx, c=c, hw=hw, kids=[], mass=m[idx].sum())
        nodes.append(node)
        if len(idx) > cap:
            code = (X[idx] >= c) @ np.array([1, 2, 4])
            for o in range(8):
                s = np.array([1.0 if o >> a & 1 else -1.0 for a in range(3)])
                node["kids"].append(build(idx[code == o], c + s * 0.5 * hw, 0.5 * hw))
        return k

    build(np.arange(len(X)), 0.5 * (lo + hi), 1.0001 * max(0.5 * (hi - lo).max(), EPS + 1e-6))
    return nodes


def taylor_force(d0, delta, m, order):
    """Sum over bodies of m f(d0 + delta), f(d) = d (|d|^2 + eps^2)^-1.5, to the given order in
    delta; d0 (T, 3), delta (B, 3).  Also the sum of the magnitudes of the order-0 terms."""
    s0 = (d0 ** 2).sum(1)[:, None] + EPS * EPS
    b, c = d0 @ delta.T, (delta ** 2).sum(1)[None]
    u = [s0 ** -1.5 + 0 * b]  # u(t) = (s0 + 2 b t + c t^2)^-1.5: s u' = -1.5 s' u
    for k in range(order):
        acc = -1.5 * (2 * b * u[k] + (2 * c * u[k - 1] if k else 0))
        acc = acc - 2 * b * k * u[k] - (c * (k - 1) * u[k - 1] if k else 0)
        u.append(acc / (s0 * (k + 1)))
    head = sum(u[: order + 1])
    tail = sum(u[:order]) if order else 0 * b
    f = (m * head).sum(1)[:, None] * d0 + (m * tail) @ delta
    return f, np.linalg.norm((m * u[0]).sum(1)[:, None] * d0, axis=1)


def expected(X, m, cap, order):
    nodes = octree(X, m, cap)
    A, mag = np.zeros_like(X), np.zeros(len(X))
    for t in (n for n in nodes if not n["kids"] and n["mass"] > 0):
        stack = [0]
        while stack:
            s = nodes[stack.pop()]
            if s["mass"] <= 0:
                continue
            dist = np.linalg.norm(s["c"] - t["c"])
            if s is not t and dist > 0 and 2.0 * (t["hw"] + s["hw"]) / dist < THETA:
                com = (m[s["idx"], None] * X[s["idx"]]).sum(0) / s["mass"]
                f, g = taylor_force(com - X[t["idx"]], X[s["idx"]] - com, m[s["idx"]], order)
            elif not s["kids"]:
                d = X[s["idx"]][None] - X[t["idx"]][:, None]
                w = m[s["idx"]] * ((d ** 2).sum(2) + EPS * EPS) ** -1.5
                f, g = (w[..., None] * d).sum(1), (w * np.linalg.norm(d, axis=2)).sum(1)
            else:
                stack += s["kids"]
                continue
            A[t["idx"]] += f
            mag[t["idx"]] += g
    return A, mag


@pytest.mark.parametrize("n,cap,cluster", [(400, 1, 0), (500, 2, 0), (600, 3, 0), (800, 5, 0), (1200, 9, 0),
                                           (2000, 33, 0), (2500, 64, 0), (900, 300, 200)])
@pytest.mark.parametrize("order", [0, 2, 4])
def test_far_field(n, cap, cluster, order):
    rng = np.random.default_rng(n + cap)
    X = rng.uniform(-2.0, 2.0, (n, 3))
    if cluster:  # leaves above a block of targets, far from the rest
        X[:cluster] = [9.0, 9.0, 9.0] + 0.1 * rng.standard_normal((cluster, 3))
    m = rng.uniform(0.1, 1.0, n)
    ref, mag = expected(X, m, cap, order)
    x, y, z = (np.ascontiguousarray(v) for v in X.T)
    for precision, tol in (("f64", 1e-11), ("mixed", 1e-5)):
        a = [np.zeros(n) for _ in range(3)]
        gx.fmm.fmm_accelerations(x, y, z, m, *a, gx.PhysicsParams(1.0, EPS),
                                 gx.FmmOptions(theta=THETA, leaf_capacity=cap, expansion_order=order), precision)
        assert (np.linalg.norm(np.stack(a, 1) - ref, axis=1) / mag).max() <= tol, precision
