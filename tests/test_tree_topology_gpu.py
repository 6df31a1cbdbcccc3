"""Octree topology from sorted keys (B200): the host builder's leaves and lists.

Sizes below, at and above a block of 1024 bodies and the 32 blocks that a lane scans one of, leaves of
one body and of more than all, shallow trees (max_depth), bodies that share cells down to the last
level, and the number of levels that sessions sort.
"""
import numpy as np
import pytest

import gx

pytestmark = pytest.mark.gpu


def system(n, kind):
    p = gx.ics.two_disk_encounter(max(1, n - n // 2), n // 2, 70 + n, 0.02)
    if kind == "clump" and n > 64:  # a deep branch: 40 bodies within 1e-5 of each other
        rng = np.random.default_rng(n)
        for f in ("x", "y", "z"):
            getattr(p, f)[20:60] = getattr(p, f)[20] + 1e-5 * rng.standard_normal(40)
    if kind == "line":  # one octant path: every split leaves most octants empty
        p.x[:] = np.linspace(0.0, 1.0, n) ** 3
        p.y[:] = p.x
        p.z[:] = p.x
    return p


@pytest.mark.parametrize("n", [1, 2, 31, 1000, 1024, 1025, 33000, 70001])
@pytest.mark.parametrize("cap", [1, 16, 100000])
@pytest.mark.parametrize("kind", ["disks", "clump", "line"])
def test_device_tree_equals_the_host_builders(n, cap, kind):
    p = system(n, kind)
    n_near = 0
    for depth in (32, 3):
        if cap == 1 and n > 2000 and (depth == 3 or kind == "line"):
            continue  # near lists of most of the system
        host = gx.build_leaf_lists(p.x, p.y, p.z, p.m, 0.02, 0.6, cap, max_depth=depth)
        dev = gx.build_leaf_lists(p.x, p.y, p.z, p.m, 0.02, 0.6, cap, max_depth=depth, on_device=True)
        for f in ("leaf_offsets", "leaf_particles", "near_offsets", "near_leaves"):
            assert np.array_equal(getattr(host, f), getattr(dev, f)), (f, depth)
        assert (host.n_far, host.n_pairs) == (dev.n_far, dev.n_pairs)


@pytest.mark.parametrize("n,cap", [(1000, 16), (33000, 64)])
def test_session_levels(n, cap):
    """A session sorts two levels more than its first tree had; a clump that forms later needs more."""
    params, opt = gx.PhysicsParams(1.0, 0.02), gx.FmmOptions(theta=0.6, leaf_capacity=cap)
    p = system(n, "disks")
    q = system(n, "clump")
    with gx.Session(n, params) as s:
        s.set_fmm(opt)
        for r in (p, q):
            s.set_state(r.x, r.y, r.z, r.vx, r.vy, r.vz, r.m)
            s.compute_accelerations("f64")
            s.step(2, 0.0, "f64")
            st = s.get_state()
            a = [np.zeros(n) for _ in range(3)]
            gx.fmm.fmm_accelerations(r.x, r.y, r.z, r.m, *a, params, opt, "f64")
            scale = np.linalg.norm(np.stack(a), axis=0).max()
            for f, v in zip(("ax", "ay", "az"), a):
                assert np.abs(st[f] - v).max() <= 1e-12 * scale
