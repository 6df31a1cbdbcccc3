"""The default variant and source split on both sides of every line of their rules (B200).

FP64 changes shape at 1500 and 15,000 targets (6000 without softening) and mixed splits change at
7000 and 18,000 sources; few targets against many sources shorten the chunks.  Tolerances of the
forms: FP64 1e-11 relative, mixed median 1e-6 and 1e-4 at most.
"""
import numpy as np
import pytest

import gx
import oracle
from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1499, 1500, 5999, 6000, 6999, 7000, 14999, 15000, 17999, 18000])
@pytest.mark.parametrize("eps", [0.02, 0.0])
def test_default_choice(n, eps):
    p = gx.ics.two_disk_encounter(n - n // 2, n // 2, n, 0.02)
    idx = np.unique(np.linspace(0, n - 1, 97).astype(np.int64))
    ref = oracle.direct_indexed(p.x, p.y, p.z, p.m, 1.0, eps, idx)
    for prec in (gx.PRECISION_F64, gx.PRECISION_MIXED):
        q = p.copy()
        gx.compute_cuda_direct_accelerations(q, gx.PhysicsParams(1.0, eps), prec)
        e = rel_err(q.accelerations[idx], ref)
        if prec == gx.PRECISION_F64:
            assert e.max() <= 1e-11
        elif eps > 0.0:
            assert np.median(e) <= 1e-6 and e.max() <= 1e-4
        else:  # close pairs amplify FP32 offset rounding without softening: the bulk only
            assert np.median(e) <= 1e-5


@pytest.mark.parametrize("targets", [1, 63, 700, 1501])
def test_few_targets_many_sources(targets):
    n = 20011
    p = gx.ics.two_disk_encounter(n - n // 2, n // 2, 5, 0.02)
    params = gx.PhysicsParams(1.0, 0.02)
    idx = np.random.default_rng(targets).choice(n, targets, replace=False)
    ref = oracle.direct_indexed(p.x, p.y, p.z, p.m, 1.0, 0.02, idx)
    assert rel_err(gx.indexed_accelerations(p, params, idx, gx.PRECISION_F64), ref).max() <= 1e-11
    e = rel_err(gx.indexed_accelerations(p, params, idx, gx.PRECISION_MIXED), ref)
    assert np.median(e) <= 1e-6 and e.max() <= 1e-4
