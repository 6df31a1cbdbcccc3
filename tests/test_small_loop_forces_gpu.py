"""FP64 step loop of small systems: accelerations, velocities and positions at the edges of its passes and
in every shape (B200).

After any number of steps the accelerations are those of the loop's own final positions, so they are
compared with the oracle's sum there.  A sum of n terms in any order, each term within 4 units of
rounding, is within (terms added one after the other + 8) * 2^-53 * sum |terms| of the exact one; at
most n / 8 terms follow one another in a lane or thread, and the reference adds all n.
"""
import numpy as np
import pytest

import gx
import oracle

pytestmark = pytest.mark.gpu

F64 = gx.PRECISION_F64
U = 2.0 ** -53


def sums_of_magnitudes(x, m, eps):
    """sum_j m_j |d| s^-3/2 per body and component, x (3, n)."""
    out = np.empty_like(x)
    for i in range(x.shape[1]):
        d = x - x[:, i:i + 1]
        s = (d * d).sum(0) + eps * eps
        w = np.where(s > 0.0, m / np.where(s > 0.0, s, 1.0) ** 1.5, 0.0)
        out[:, i] = (np.abs(d) * w).sum(1)
    return out


def run(p, eps, steps, dt, persistent):
    with gx.Session(len(p), gx.PhysicsParams(1.0, eps)) as s:
        s.set_persistent(persistent)
        s.set_particles(p)
        s.compute_accelerations(F64)
        s.step(steps, dt, F64)
        return s.get_state()


@pytest.fixture
def shape():
    def force(tpw, wpt):
        gx._ffi.call("gx_debug_small_targets_per_warp", tpw)
        gx._ffi.call("gx_debug_small_warps_per_target", wpt)
    yield force
    force(0, 0)


SIZES = [2, 33, 255, 1023, 1024, 1025, 1056, 2047, 2048, 2049, 3073, 4096]
FORCED = [(n, tpw, wpt) for n in (33, 1023, 1025, 2049) for tpw in (1, 2, 4) for wpt in (1, 2)]


@pytest.mark.parametrize("eps", [0.05, 0.0])
@pytest.mark.parametrize("n,tpw,wpt", [(n, 0, 0) for n in SIZES] + FORCED)
def test_forces_of_the_final_positions(n, eps, tpw, wpt, shape):
    p = gx.ics.two_disk_encounter(n - n // 2, n // 2, 900 + n, 0.05)
    p.m[::5] *= 1e-3  # light sources count as well as heavy ones only where the terms are weighed
    shape(tpw, wpt)
    steps, dt = 3, 1e-3
    st = run(p, eps, steps, dt, True)
    shape(0, 0)
    x = np.stack([st[f] for f in ("x", "y", "z")])
    mag = sums_of_magnitudes(x, p.m, eps)
    ref = oracle.direct_targets(*x, p.m, 1.0, eps).T
    got = np.stack([st[f] for f in ("ax", "ay", "az")])
    bound = (n + n / 8 + 32) * U * mag
    assert np.all(np.abs(got - ref) <= bound)
    # the loop of launches takes the same steps: its kicks differ by the sums' rounding only
    other = run(p, eps, steps, dt, False)
    for c, f in enumerate(("x", "y", "z")):
        vel = steps * dt * bound[c].max() * 8 + 8 * U * np.abs(st["v" + f]).max()
        assert np.abs(st["v" + f] - other["v" + f]).max() <= vel
        assert np.abs(st[f] - other[f]).max() <= steps * dt * vel + 8 * U * np.abs(st[f]).max()
        if eps > 0.0:  # two positions a rounding apart: |da| <= 4 sum m / eps^3 |dx|
            apart = 4.0 * p.m.sum() / eps ** 3 * (steps * dt * vel + 8 * U * np.abs(st[f]).max())
            assert np.abs(st["a" + f] - other["a" + f]).max() <= 2 * bound[c].max() + 3 * apart
