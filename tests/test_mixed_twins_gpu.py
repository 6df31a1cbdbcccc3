"""Mixed variants with the same tiles over other threads give the same bits (B200)."""
import numpy as np
import pytest

import gx

pytestmark = pytest.mark.gpu
MIX = gx.PRECISION_MIXED


def variants():
    out = {}
    for v in range(64):
        try:
            out[v] = gx.describe_variant(MIX, v)
        except gx.GxError:
            continue
    return out


@pytest.mark.parametrize("shapes", [("block=256 ipt=4 jt=512 f32x2-targets", "block=512 ipt=2 jt=512 f32x2-targets"),
                                    ("block=64 ipt=4 jt=256 f32x2", "block=256 ipt=1 jt=256 f32x2")])
@pytest.mark.parametrize("n,js", [(3, 1), (255, 1), (257, 1), (1025, 2), (5000, 3), (7003, 7)])
def test_twins_are_bit_identical(shapes, n, js):
    ids = [next(v for v, d in variants().items() if d == "mixed " + s) for s in shapes]
    p = gx.ics.two_disk_encounter(n - n // 2, n // 2, n, 0.02)
    got = []
    with gx.Session(n, gx.PhysicsParams(1.0, 0.02)) as s:
        s.set_particles(p)
        for v in ids:
            s.set_config(MIX, v, js)
            s.compute_accelerations(MIX)
            st = s.get_state()
            got.append(np.stack([st["ax"], st["ay"], st["az"]]))
    assert np.array_equal(got[0], got[1])
