"""FP64 sums without softening at pairs whose weight overflows (B200).

|d|^2 from 1e-216 to 1e-204: 1 / |d|^3 is infinite or nearly, and the reference's sum over such
sources is infinite with the sign of the offset (NaN where signs meet or an offset is zero).
"""
import numpy as np
import pytest
import torch

import gx
import oracle

pytestmark = pytest.mark.gpu

F64 = gx.PRECISION_F64
PARAMS = gx.PhysicsParams(1.0, 0.0)


def cluster(n):
    """Body 0 at the origin, 40 within 1e-108 to 1e-103 of it, the rest far away."""
    p = gx.ics.two_disk_encounter(n - n // 2, n // 2, n, 0.05)
    rng = np.random.default_rng(n)
    d = rng.uniform(0.3, 1.0, (3, 40)) * 10.0 ** rng.uniform(-107.5, -103.0, 40)
    for c, f in enumerate(("x", "y", "z")):
        a = getattr(p, f)
        a += 2.0
        a[0] = 0.0
        a[1:41] = d[c]
    p.m[7] = 0.0
    return p


def kinds(a):
    a = np.asarray(a)
    return np.where(np.isnan(a), 2, np.where(np.isposinf(a), 1, np.where(np.isneginf(a), -1, 0)))


@pytest.mark.parametrize("n", [64, 300, 2000, 9001])
def test_direct_sum_overflows_as_the_reference(n):
    p = cluster(n)
    with np.errstate(all="ignore"):
        ref = oracle.direct_targets(p.x, p.y, p.z, p.m, 1.0, 0.0)
    q = p.copy()
    gx.compute_cuda_direct_accelerations(q, PARAMS, F64)
    got = q.accelerations
    assert np.all(np.isposinf(got[0])) and np.array_equal(kinds(got)[1:41] == 0, kinds(ref)[1:41] == 0)
    far = np.r_[41:n]
    scale = np.linalg.norm(ref[far], axis=1, keepdims=True)
    assert np.all(np.abs(got[far] - ref[far]) <= 1e-11 * scale)


def test_step_loop_and_near_field_overflow_too():
    n = 300
    p = cluster(n)
    with gx.Session(n, PARAMS) as s:
        s.set_particles(p)
        s.step(1, 0.0, F64)
        st = s.get_state()
    assert all(np.isposinf(st[f][0]) for f in ("ax", "ay", "az"))
    lists = gx.fmm_p2p.LeafLists(np.array([0, n], np.int32), np.arange(n, dtype=np.int32), np.array([0, 1], np.int32),
                                 np.zeros(1, np.int32))
    acc = [np.zeros(n) for _ in range(3)]
    gx.fmm_p2p.p2p_leaves(p.x, p.y, p.z, p.m, lists, PARAMS, *acc, F64)
    assert all(np.isposinf(a[0]) for a in acc)
