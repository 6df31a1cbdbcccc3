"""Interaction lists made in one walk (B200): lists, statistics and accelerations at the edges.

Near lists shorter and longer than the walk's buffer (512) and sorted in registers by 1 to 16
values per lane, far lists of none, part of and several chunks of 512, target ranges, and -- with
gx_debug_fmm_tight_pools -- pools that are too small at first and a stack of 64 entries, so that
leaves overflow it.  The host builder's lists are the reference's; a far list in another order
changes only the rounding of the far field's sums (at most a few thousand terms: 1e-12).
"""
import numpy as np
import pytest

import gx

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[False, True], ids=["pools", "tight"])
def tight(request):
    gx._ffi.call("gx_debug_fmm_tight_pools", 2 if request.param else 0)
    yield request.param
    gx._ffi.call("gx_debug_fmm_tight_pools", 0)


CASES = [(1, 16, 0.6), (9, 1, 0.6), (300, 4, 0.6), (2000, 1, 0.3), (6000, 8, 0.35), (20000, 64, 0.6), (30000, 16, 0.5)]


@pytest.mark.parametrize("n,cap,theta", CASES)
def test_lists_equal_the_host_builders(n, cap, theta, tight):
    p = gx.ics.two_disk_encounter(n - n // 2, n // 2, 40 + n, 0.02)
    if n > 100:
        p.m[5::9] = 0.0  # massless bodies and leaves
    host = gx.build_leaf_lists(p.x, p.y, p.z, p.m, 0.02, theta, cap)
    dev = gx.build_leaf_lists(p.x, p.y, p.z, p.m, 0.02, theta, cap, on_device=True)
    assert dev.built_on_device
    for f in ("leaf_offsets", "leaf_particles", "near_offsets", "near_leaves"):
        assert np.array_equal(getattr(host, f), getattr(dev, f)), f
    assert (host.n_far, host.n_pairs) == (dev.n_far, dev.n_pairs)


@pytest.mark.parametrize("n,cap,theta", CASES)
def test_accelerations_with_tight_pools(n, cap, theta):
    p = gx.ics.two_disk_encounter(n - n // 2, n // 2, 50 + n, 0.02)
    params, opt = gx.PhysicsParams(1.0, 0.02), gx.FmmOptions(theta=theta, leaf_capacity=cap)
    got = []
    for tight in (0, 2):
        gx._ffi.call("gx_debug_fmm_tight_pools", tight)
        try:
            q = p.copy()
            s = gx.FastMultipoleSolver(params, opt)
            s.compute(q)
            r = p.copy()
            r.ax[:] = 7.0
            gx.compute_fmm_accelerations_for_targets(r, params, n // 3, n - n // 4, opt)
            got.append((q.accelerations, s.stats(), r))
        finally:
            gx._ffi.call("gx_debug_fmm_tight_pools", 0)
    assert got[0][1] == got[1][1]
    scale = np.linalg.norm(got[0][0], axis=1).max() + 1e-300
    assert np.abs(got[0][0] - got[1][0]).max() <= 1e-12 * scale
    lo, hi = n // 3, n - n // 4
    for a, _, r in got:
        assert np.abs(r.accelerations[lo:hi] - a[lo:hi]).max(initial=0.0) <= 1e-12 * scale
        assert np.all(r.ax[:lo] == 7.0) and np.all(r.ax[hi:] == 7.0)
