"""Step loop of small systems at the edges of its passes (B200): 512 sources (exact form) and 1024
(FP64), one, two and four targets per warp, against the loop of single launches -- the exact form bit
for bit, FP64 within 1e-12 -- with close pairs that the exact reciprocal leaves to IEEE division.
"""
import numpy as np
import pytest

import gx

pytestmark = pytest.mark.gpu

EXACT, F64 = gx.PRECISION_F64_EXACT, gx.PRECISION_F64


@pytest.mark.parametrize("n", [1, 31, 32, 33, 511, 512, 513, 545, 1023, 1024, 1025, 2047, 2049, 3071, 4095])
@pytest.mark.parametrize("eps", [0.05, 0.0])
def test_loop_equals_launches(n, eps):
    p = gx.ics.two_disk_encounter(n - n // 2, n // 2, 300 + n, 0.05)
    if n > 40:
        p.x[7], p.y[7], p.z[7] = p.x[8], p.y[8], p.z[8]            # a coincident pair
        p.x[30] = p.x[31] + 1e-200                                 # and one below the fast range
        p.y[30], p.z[30] = p.y[31], p.z[31]
        p.m[n // 2] = 0.0
    got = {}
    for persistent in (True, False):
        for prec in (EXACT, F64):
            with gx.Session(n, gx.PhysicsParams(1.0, eps)) as s:
                s.set_persistent(persistent)
                s.set_particles(p)
                s.compute_accelerations(prec)
                s.step(3, 1e-4, prec)
                got[persistent, prec] = s.get_state()
    for f in ("x", "y", "z", "vx", "vy", "vz", "ax", "ay", "az"):
        assert np.array_equal(got[True, EXACT][f], got[False, EXACT][f], equal_nan=True), f
    if eps > 0.0:
        for f in ("x", "y", "z"):
            assert np.abs(got[True, F64][f] - got[False, F64][f]).max() <= 1e-12
