"""Node moments bit for bit against a restatement in plain doubles (B200).

Trees of one leaf (the edges of the 32-body staging) and of one split (a root over eight leaves,
some of them empty or massless): P2M and M2M as the reference orders their operations
(cpp/fmm/multipole.cpp:218-252, cpp/fmm/fmm_solver.cpp:157-208), in Python floats, which round
every operation once as the reference's build does.
"""
import ctypes
import math

import numpy as np
import pytest

import gx

pytestmark = pytest.mark.gpu

EXPONENTS = [(x, y, d - x - y) for d in range(5) for x in range(d, -1, -1) for y in range(d - x, -1, -1)]


def power(v, e):
    r = 1.0
    for _ in range(e):
        r *= v
    return r


def leaf_record(bodies, cell):
    mass = wx = wy = wz = 0.0
    for x, y, z, m in bodies:
        mass += m
        wx += x * m
        wy += y * m
        wz += z * m
    com = (wx / mass, wy / mass, wz / mass) if mass > 0.0 else cell
    mom = []
    for ex, ey, ez in EXPONENTS[4:]:
        v = 0.0
        for x, y, z, m in bodies:
            v += m * (power(x - com[0], ex) * power(y - com[1], ey) * power(z - com[2], ez))
        mom.append(v)
    return [*com, mass, *mom]


def parent_record(children):
    mass = wx = wy = wz = 0.0
    for c in children:
        if c[3] > 0.0:
            mass += c[3]
            wx += c[0] * c[3]
            wy += c[1] * c[3]
            wz += c[2] * c[3]
    com = (wx / mass, wy / mass, wz / mass)
    total = [0.0] * 31
    for c in children:
        if not c[3] > 0.0:
            continue
        s = [c[k] - com[k] for k in range(3)]
        for a, alpha in enumerate(EXPONENTS[4:]):
            value = 0.0
            for b, beta in enumerate(EXPONENTS):
                if any(beta[k] > alpha[k] for k in range(3)) or sum(beta) == 1:
                    continue
                binom = 1.0
                for k in range(3):
                    binom *= math.comb(alpha[k], beta[k])
                sf = binom * power(s[0], alpha[0] - beta[0]) * power(s[1], alpha[1] - beta[1]) * power(s[2], alpha[2] - beta[2])
                if sf != 0.0:
                    value += sf * (c[3] if b == 0 else c[b])
            total[a] += value
    return [*com, mass, *total]


def engine_records(x, y, z, m, cap):
    opt = gx.FmmOptions(leaf_capacity=cap).ffi()
    phys = gx.PhysicsParams(1.0, 0.02).ffi()
    n = ctypes.c_int64()
    args = [len(x), *(gx._ffi.ptr(v) for v in (x, y, z, m)), phys, opt]
    gx._ffi.call("gx_fmm_moments", *args, 0, None, ctypes.byref(n))
    rec = np.empty((n.value, 35))
    gx._ffi.call("gx_fmm_moments", *args, n.value, gx._ffi.ptr(rec), ctypes.byref(n))
    return rec


def bodies(n, seed):
    rng = np.random.default_rng(seed)
    return [rng.uniform(-3.0, 5.0, n) for _ in range(3)] + [rng.uniform(0.1, 2.0, n)]


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 97])
def test_one_leaf(n):
    x, y, z, m = bodies(n, n)
    rec = engine_records(x, y, z, m, 128)
    assert rec.shape[0] == 1
    assert np.array_equal(rec[0], leaf_record(list(zip(x.tolist(), y.tolist(), z.tolist(), m.tolist())), None))


@pytest.mark.parametrize("n,octants,massless", [(40, 8, 0), (130, 8, 3), (90, 3, 0), (300, 5, 2)])
def test_one_split(n, octants, massless):
    x, y, z, m = bodies(n, 7 * n)
    # corners fix the root cell at (-4, 4)^3 (up to its margin); the others stay in some octants
    o = np.arange(n) % octants
    for c, v in enumerate((x, y, z)):
        v[:] = np.where(o >> c & 1, 1.0, -1.0) * (0.5 + 3.0 * np.random.default_rng(n + c).random(n))
        v[0], v[octants - 1] = -4.0, np.where((octants - 1) >> c & 1, 4.0, v[octants - 1])
    m[o < massless] = 0.0
    rec = engine_records(x, y, z, m, max(n // octants + 1, 1))
    lo = [v.min() for v in (x, y, z)]
    hi = [v.max() for v in (x, y, z)]
    centre = [(a + b) * 0.5 for a, b in zip(lo, hi)]
    octant = sum((v >= c).astype(int) << k for k, (v, c) in enumerate(zip((x, y, z), centre)))
    kids = []
    for k in range(8):
        sel = np.flatnonzero(octant == k)
        assert len(sel) <= n // octants + 1
        kids.append(leaf_record([(float(x[i]), float(y[i]), float(z[i]), float(m[i])) for i in sel], (0.0, 0.0, 0.0)))
    want = [parent_record(kids)] + [k for k in kids if k[3] > 0.0]
    assert np.array_equal(rec, np.array(want))
