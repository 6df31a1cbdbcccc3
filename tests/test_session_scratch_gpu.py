"""Partial sums of a session's split direct sums (B200)."""
import numpy as np
import pytest
import torch

import gx
import oracle
from conftest import rel_err

pytestmark = pytest.mark.gpu

F64, MIX = gx.PRECISION_F64, gx.PRECISION_MIXED
PART_LIMIT = 256 << 20  # what the partial sums of one evaluation may take


@pytest.mark.parametrize("prec", [F64, MIX])
def test_scratch_follows_the_targets(prec):
    """A rank's range of a larger system: the scratch is that of its own targets (an FP64 evaluation
    takes many source chunks), and a larger range set later still fits."""
    n, count = 1 << 18, 1 << 14
    p = gx.ics.two_disk_encounter(n // 2, n // 2, 23, 0.02)
    idx = np.arange(5, count, count // 40)
    with gx.Session(n, gx.PhysicsParams(1.0, 0.02)) as s:
        s.set_particles(p)
        s.synchronize()
        s.set_targets(n // 4, count)
        free = torch.cuda.mem_get_info()[0]
        s.compute_accelerations(prec)
        s.synchronize()
        used = free - torch.cuda.mem_get_info()[0]
        js = s.get_config(prec)[1]
        assert used <= 24 * js * count + 4 * (n // 64 + 1) + (4 << 20) and used <= PART_LIMIT
        s.set_targets(n // 4 + 1, 2 * count + 1)
        s.compute_accelerations(prec)
        st = s.get_state()
    ref = oracle.direct_indexed(p.x, p.y, p.z, p.m, 1.0, 0.02, n // 4 + 1 + idx)
    got = np.stack([st[f][n // 4 + 1 + idx] for f in ("ax", "ay", "az")], 1)
    e = rel_err(got, ref)
    if prec == F64:
        assert e.max() <= 1e-11
    else:
        assert np.median(e) <= 1e-6 and e.max() <= 1e-4


@pytest.mark.parametrize("n", [20000, 40001])
def test_recorded_steps_follow_the_scratch(n):
    """Steps recorded before the scratch grew (FP64 takes more chunks than mixed) run with the new one:
    the same bits as in a session whose scratch was large from the start, and nothing is written to
    memory that somebody else holds by then."""
    p = gx.ics.two_disk_encounter(n - n // 2, n // 2, 29, 0.05)
    out = []
    for large_first in (True, False):
        with gx.Session(n, gx.PhysicsParams(1.0, 0.05)) as s:
            if large_first:
                s.set_particles(p)
                s.compute_accelerations(F64)
            s.set_particles(p)
            s.compute_accelerations(MIX)
            s.step(2, 0.002, MIX)
            s.compute_accelerations(F64)
            s.synchronize()
            torch.cuda.empty_cache()
            held = [torch.full((k << 18,), 7.0, dtype=torch.float64, device="cuda") for k in (1, 2, 4, 8)]
            torch.cuda.synchronize()
            s.step(2, 0.002, MIX)
            out.append(s.get_state())
            assert all(bool((t == 7.0).all()) for t in held)
    for f in out[0]:
        assert np.array_equal(out[0][f], out[1][f]), f
