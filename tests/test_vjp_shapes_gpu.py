"""The adjoint kernels at the edges of their tiles, shapes and splits (B200), against FP64 torch.

FP64: sums of n terms of mixed sign, 1e-12 of the largest gradient; mixed: FP32 pair terms, 2e-5
of it (the maximum over bodies of errors whose median is a few 1e-7).
"""
import pytest

import gx
from gx.adjoint import direct_vjp

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def torch_vjp(X, m, lam, eps):
    d = X[:, None, :] - X[:, :, None]
    s = (d * d).sum(0) + eps * eps
    i3 = torch.where(s > 0, s, torch.ones_like(s)) ** -1.5
    i3 = torch.where(s > 0, i3, torch.zeros_like(s))
    i5 = torch.where(s > 0, i3 / torch.where(s > 0, s, torch.ones_like(s)), torch.zeros_like(s))
    A = m[None, :, None] * lam[:, None, :] - m * lam[:, :, None]
    g = (A * i3 - 3.0 * d * (i5 * (A * d).sum(0))).sum(2)
    return g, -(i3 * (d * lam[:, None, :]).sum(0)).sum(1)


@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 127, 129, 255, 257, 511, 513, 1000, 3001])
@pytest.mark.parametrize("eps", [0.05, 0.0])
def test_sizes(n, eps):
    p = gx.ics.two_disk_encounter(n - n // 2, n // 2, n, 0.05)
    X = torch.tensor(p.positions.T.copy(), device="cuda")
    m = torch.tensor(p.m, device="cuda")
    lam = torch.randn(3, n, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(n))
    params = gx.PhysicsParams(1.0, eps)
    want = torch_vjp(X, m, lam, eps)
    for prec, tol in ((gx.PRECISION_F64, 1e-12), (gx.PRECISION_MIXED, 2e-5)):
        if prec == gx.PRECISION_MIXED and eps == 0.0:
            continue  # close pairs amplify FP32 offset rounding without softening
        for got, ref in zip(direct_vjp(X, m, lam, params, prec), want):
            assert torch.all((got - ref).abs() <= tol * ref.abs().max() + 1e-300)


@pytest.mark.parametrize("n", [11999, 12000])
def test_fp64_shapes_agree(n):
    p = gx.ics.two_disk_encounter(n - n // 2, n // 2, 3, 0.05)
    X = torch.tensor(p.positions.T.copy(), device="cuda")
    m = torch.tensor(p.m, device="cuda")
    lam = torch.randn(3, n, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    got = direct_vjp(X, m, lam, gx.PhysicsParams(1.0, 0.05), gx.PRECISION_F64)
    # the first 500 targets against all sources
    d = X[:, None, :] - X[:, :500, None]
    s = (d * d).sum(0) + 0.05 * 0.05
    A = m[None, :500, None] * lam[:, None, :] - m * lam[:, :500, None]
    g = (A * s**-1.5 - 3.0 * d * (s**-2.5 * (A * d).sum(0))).sum(2)
    h = -(s**-1.5 * (d * lam[:, None, :]).sum(0)).sum(1)
    for a, b in ((got[0][:, :500], g), (got[1][:500], h)):
        assert torch.all((a - b).abs() <= 1e-12 * b.abs().max())
