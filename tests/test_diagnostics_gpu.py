"""Diagnostics of a resident session at the edges of the kernel's tiles (B200).

Every unordered pair is taken once over tiles of 64 bodies (up to 8192) or 256 (above), in
double rows of tiles; sizes below, at and above the tile edges, odd and even tile counts.
Sums of up to n^2 / 2 positive terms in FP64: 1e-12 of the value (the momentum and the centre of
mass cancel, so they are compared on the scale of the sums of their magnitudes).
"""
import numpy as np
import pytest

import gx
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 129, 1000, 8191, 8192, 8193, 8448, 8705])
def test_session_diagnostics_at_tile_edges(n):
    eps = 0.03
    p = gx.ics.two_disk_encounter(n - n // 2, n // 2, 100 + n, eps, mass2=0.5)
    ref = np.array(oracle.diagnostics(p.x, p.y, p.z, p.vx, p.vy, p.vz, p.m, 1.0, eps))
    scale = np.abs(ref).copy()
    X, V = p.positions, p.velocities
    scale[4:7] = np.abs(V * p.m[:, None]).sum(0)
    scale[7:10] = np.abs(X * p.m[:, None]).sum(0) / p.m.sum()
    scale[10:13] = (np.abs(X).max(1) * np.abs(V).max(1) * p.m).sum() * 2
    with gx.Session(n, gx.PhysicsParams(1.0, eps)) as s:
        s.set_particles(p)
        rows = [np.array(s.diagnostics().as_row()) for _ in range(3)]
    assert np.array_equal(rows[0], rows[1]) and np.array_equal(rows[0], rows[2])
    assert np.all(np.abs(rows[0] - ref) <= 1e-12 * np.maximum(scale, np.abs(ref)) + 1e-300)
