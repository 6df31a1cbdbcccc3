"""A session that owns no bodies (a rank beyond the last body) takes every call (B200).

Nothing is kicked, drifted or given a force, so the whole state stays as it was set, and a range set
afterwards evaluates as usual.
"""
import numpy as np
import pytest

import gx

pytestmark = pytest.mark.gpu

FIELDS = ("x", "y", "z", "vx", "vy", "vz", "ax", "ay", "az")


@pytest.mark.parametrize("prec", [gx.PRECISION_F64, gx.PRECISION_MIXED, gx.PRECISION_F64_EXACT])
@pytest.mark.parametrize("n,eps", [(700, 0.05), (700, 0.0), (20000, 0.05)])
def test_calls_without_targets(prec, n, eps):
    p = gx.ics.two_disk_encounter(n // 2, n // 2, 17, 0.05)
    rng = np.random.default_rng(4)
    p.ax, p.ay, p.az = rng.normal(size=(3, n))
    with gx.Session(n, gx.PhysicsParams(1.0, eps)) as s:
        s.set_particles(p)
        s.set_state(p.x, p.y, p.z, p.vx, p.vy, p.vz, p.m, p.ax, p.ay, p.az)
        for begin in (0, n // 3, n):
            s.set_targets(begin, 0)
            s.compute_accelerations(prec)
            s.step(3, 0.01, prec)
            s.kick_drift(0.01, 0.01)
            s.force_kick(0.01, prec)
            variant, jsplit = s.get_config(prec)
            assert variant >= 0 and jsplit == 1
            s.autotune(prec)
            s.compute_accelerations(prec)
            st = s.get_state()
            for f in FIELDS:
                assert np.array_equal(st[f], getattr(p, f)), f
        s.set_targets(n // 3, n // 2)
        s.compute_accelerations(prec)
        st = s.get_state()
    q = p.copy()
    b, e = n // 3, n // 3 + n // 2
    gx.compute_direct_accelerations_for_targets(q, gx.PhysicsParams(1.0, eps), b, e, prec)
    for f in ("ax", "ay", "az"):
        assert np.array_equal(st[f][:b], getattr(p, f)[:b]) and np.array_equal(st[f][e:], getattr(p, f)[e:])
        scale = np.abs(getattr(q, f)[b:e]).max()
        tol = 0.0 if prec == gx.PRECISION_F64_EXACT else 1e-12 if prec == gx.PRECISION_F64 else 1e-4
        assert np.abs(st[f][b:e] - getattr(q, f)[b:e]).max() <= tol * scale
