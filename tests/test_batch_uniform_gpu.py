"""Mixed batches of equal instances whose whole tiles fill the SMs evenly (B200).

Such instances are not cut into source chunks: their sums have the bits of an unsplit evaluation of one
system with tiles of 1536 targets, while an uneven number of tiles is cut (and agrees within the
form's tolerance: median 1e-6, 1e-4 at most).
"""
import numpy as np
import pytest

import gx
from conftest import rel_err

pytestmark = pytest.mark.gpu

MIX = gx.PRECISION_MIXED
PARAMS = gx.PhysicsParams(1.0, 0.05)


def unsplit(p):
    with gx.Session(len(p), PARAMS) as s:
        s.set_particles(p)
        v = next(k for k in range(64) if gx.describe_variant(MIX, k) == "mixed block=256 ipt=6 jt=512 f32x2-targets")
        s.set_config(MIX, v, 1)
        s.compute_accelerations(MIX)
        st = s.get_state()
    return np.stack([st[f] for f in ("ax", "ay", "az")], 1)


@pytest.mark.parametrize("k,n,whole", [(148, 1536, True), (74, 1536, True), (37, 3072, True), (37, 1536, False),
                                       (16, 2000, False)])
def test_whole_tiles(k, n, whole):
    parts = [gx.ics.two_disk_encounter(n // 2, n - n // 2, 70 + i % 7, 0.05) for i in range(k)]
    cat = {f: np.concatenate([getattr(p, f) for p in parts]) for f in ("x", "y", "z", "vx", "vy", "vz", "m")}
    with gx.Batch(np.arange(k + 1) * n, PARAMS) as b:
        b.set_state(*(cat[f] for f in ("x", "y", "z", "vx", "vy", "vz", "m")))
        b.compute_accelerations(MIX)
        st = b.get_state()
    got = np.stack([st[f] for f in ("ax", "ay", "az")], 1)
    for i in {0, min(6, k - 1), k - 1}:
        ref = unsplit(parts[i])
        mine = got[i * n:(i + 1) * n]
        if whole:
            assert np.array_equal(mine, ref), i
        else:
            e = rel_err(mine, ref)
            assert np.median(e) <= 1e-6 and e.max() <= 1e-4
