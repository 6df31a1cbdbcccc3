"""List pools of a single FMM evaluation when memory is short (B200).

The pools are guessed before the lists are known.  A guess that does not fit is replaced by what the
lists need, with the same results; only a need that does not fit is an error, and the next call works.
"""
import numpy as np
import pytest
import torch

import gx
import oracle
from gx import _ffi
from conftest import rel_err

pytestmark = pytest.mark.gpu

CHUNK = 512  # far nodes per pool chunk


@pytest.fixture
def limit():
    def set_limit(n):
        _ffi.call("gx_debug_alloc_limit", int(n))
    yield set_limit
    set_limit(0)


def evaluate(p, opt, prec=gx.PRECISION_F64):
    X = [torch.from_numpy(getattr(p, f)).cuda() for f in ("x", "y", "z", "m")]
    A = [torch.zeros(len(p), dtype=torch.float64, device="cuda") for _ in range(3)]
    st = gx.fmm.fmm_accelerations(*X, *A, gx.PhysicsParams(1.0, 0.02), opt, prec)
    return st, torch.stack(A, 1).cpu().numpy()


@pytest.mark.parametrize("prec", [gx.PRECISION_F64, gx.PRECISION_MIXED])
def test_guess_that_does_not_fit(limit, prec):
    p = gx.ics.two_disk_encounter(32768, 32768, 41, 0.02)
    opt = gx.FmmOptions(theta=0.6, leaf_capacity=16)
    st, ref = evaluate(p, opt, prec)
    guess = 2 * (st.node_count - st.node_count // 8) * CHUNK * 4
    need = (st.far_interactions // CHUNK + st.leaf_count + 1) * CHUNK * 4  # at least: chunks are per leaf
    assert need < guess
    limit(need)
    st2, got = evaluate(p, opt, prec)
    assert st2 == st and np.array_equal(got, ref)
    limit(st.far_interactions)  # a quarter of the far entries' bytes
    with pytest.raises(gx.GxError) as err:
        evaluate(p, opt, prec)
    assert err.value.status == gx.GX_ERR_OUT_OF_MEMORY
    limit(0)
    st3, got = evaluate(p, opt, prec)
    assert st3 == st and np.array_equal(got, ref)


def test_single_body_leaves_take_no_more_than_the_limit(limit):
    """2^18 leaves of one body among 0.9 million cells: pools by the leaves with bodies and at most
    2 GiB each, or as much as the lists hold."""
    n = 1 << 18
    p = gx.ics.two_disk_encounter(n // 2, n // 2, 43, 0.02)
    limit(2 << 30)
    st, got = evaluate(p, gx.FmmOptions(theta=0.9, leaf_capacity=1))
    assert st.leaf_count > n // 2
    idx = np.arange(11, n, n // 50)
    e = rel_err(got[idx], oracle.direct_indexed(p.x, p.y, p.z, p.m, 1.0, 0.02, idx))
    assert np.median(e) <= 2e-2
