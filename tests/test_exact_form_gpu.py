"""The exact form's own reciprocal square root and its kernels, bit for bit against the oracle (B200).

RN(1 / RN(sqrt(s))) from fused multiply-adds could only round differently from IEEE square root
and division where the unrounded result lies within about 2^-50 ulp of a midpoint.  For the square
root these arguments are s = M^2 - d with an odd 54-bit M and a small d = M^2 mod 2^54: they are
listed here by lifting the square roots of d.  For the reciprocal they are the 53-bit divisors q of
2^106 + d (d small), listed from the factors of 2^106 + d.  Each is met as the squared distance of
a pair.
"""
import math

import numpy as np
import pytest

import gx
import oracle

pytestmark = pytest.mark.gpu
EXACT = gx.PRECISION_F64_EXACT


# 53-bit q with q (2 k + 1) = 2^106 + d for some k, |d| <= 9
HARD_DIVISORS = [
    0x1014ca35e947b6, 0x1024a3bd98da02, 0x10699d36aec84e, 0x109107683ee29e, 0x10aadc6f562fdc,
    0x10af911aa26396, 0x10d03f8a57cc76, 0x10ed85c351e224, 0x110af85de838ce, 0x110d10000221a2,
    0x1125e52b034982, 0x113deff6b41e35, 0x115efb8b10aa42, 0x11d3799c32581e, 0x11f98ea5d9b262,
    0x120a8f5bbf2106, 0x12af4d6bc06922, 0x12bf5907e316d2, 0x12d2d2d2d2d2d4, 0x12e3c6a0509ca4,
    0x12e93952a2ed6e, 0x130a0dd90e13a2, 0x132160ccc0848c, 0x134d8fe343ef42, 0x13541c0067f83c,
    0x1379cb88f092f2, 0x13a324a526d5ee, 0x13a7a1d01d1ec2, 0x13d75d54b37492, 0x1403e897077b16,
    0x14873ecade304c, 0x14a6fb45f5d782, 0x14cad5a5fa03ee, 0x15555555555554, 0x155f2490c86132,
    0x156a8cb0234262, 0x159aa11aaecb86, 0x16026c81a85766, 0x161c2909f39d4b, 0x163baaac17d1e2,
    0x163dd0554d0122, 0x16d6422e5cf246, 0x16f0f27bf434d6, 0x16fae7ba173812, 0x172f10bf899124,
    0x17641c46f799ee, 0x178cb7d5d6e322, 0x178d42e524dcdc, 0x17f52093014f0e, 0x1806c89fcb9452,
    0x181efe51ead722, 0x18401cbcdb5596, 0x184a12efef626e, 0x194ab05a4ecedc, 0x194c4511fa3124,
    0x1960a45d1a71e6, 0x199d2b42ffe9f4, 0x199e1b447e99c2, 0x19f142d24e1352, 0x1a0b8ffffcbe8e,
    0x1a149bad85de72, 0x1a2ce4d7478a06, 0x1a6f41dab98cb2, 0x1aa7c88ee59082, 0x1ae6849e786ad2,
    0x1b227794e85702, 0x1bea3278b789d2, 0x1c2693dcf34742, 0x1c36899addce3c, 0x1c384d119331c4,
    0x1c4d3aabd478f6, 0x1c69bf28eba166, 0x1c928b5b9dc714, 0x1d5b9032f086be, 0x1da210daeb138e,
    0x1de441d5331432, 0x1de4a0d00fa9b2, 0x1e20adbc4078a2, 0x1e756f08df1792, 0x1e8d517d09c5c2,
    0x1e9a9473949bf6, 0x1ef43974550f69, 0x1ef7930608393e, 0x1f65fad23b0d86, 0x1f739bd459bea2,
    0x1fe24bffeb8794, 0x1ffb8a8b628dbc, 0x1ffffff8000001, 0x1ffffffffffffd, 0x1fffffffffffff,
]


def lifted_roots(d, bits):
    """All x modulo 2^bits with x^2 = d modulo 2^bits (d = 1 modulo 8)."""
    roots = {1, 3, 5, 7}
    for b in range(4, bits + 1):
        mod = 1 << b
        roots = {y for x in roots for y in (x, x + (1 << (b - 1)), x + (1 << (b - 2))) if (y * y - d) % mod == 0}
        roots = {y % mod for y in roots}
    return roots


def hard_squares():
    """Doubles in [1, 4) whose square roots lie closest to midpoints, and neighbours of (2 - ulp)^2."""
    out = set()
    for d in range(-127, 128, 8):
        d -= (d - 1) % 8
        for x in lifted_roots(d, 54):
            for M in (x, x + (1 << 53)):
                if not (1 << 53) < M < (1 << 54) or (M * M - d) % (1 << 54):
                    continue
                s = (M * M - d) >> 54
                f = math.ldexp(float(s), -52)
                if int(float(s)) == s and 1.0 <= f < 4.0:
                    out.add(f)
    for q in HARD_DIVISORS:  # arguments whose square root rounds to q
        f = math.ldexp(float(q), -52)
        out |= {s for s in (f * f, math.nextafter(f * f, 0.0), math.nextafter(f * f, 4.0)) if math.sqrt(s) == f and s < 4.0}
    for k in range(1, 9):
        out |= {4.0 - k * 2.0**-51, 1.0 + k * 2.0**-52, 2.0 - k * 2.0**-52, 2.0 + k * 2.0**-51}
    return sorted(out)


def separation(s):
    """(y, z) with RN(RN(y y) + RN(z z)) == s."""
    y = math.sqrt(s)
    while y * y > s:
        y = math.nextafter(y, 0.0)
    z = math.sqrt(s - y * y)
    assert y * y + z * z == s
    return y, z


def system(svals, scale):
    """Body 0 at the origin; one body per value at that squared distance (times scale^2)."""
    yz = np.array([separation(s) for s in svals]) * scale
    n = len(svals) + 1
    x, y, z = np.zeros(n), np.zeros(n), np.zeros(n)
    y[1:], z[1:] = yz[:, 0], yz[:, 1]
    return x, y, z


def test_hard_squares_are_listed():
    assert len(HARD_DIVISORS) > 60 and len(hard_squares()) > 120


@pytest.mark.parametrize("scale", [1.0, 2.0**-200, 2.0**300])
def test_hard_cases_bit_for_bit(scale):
    svals = hard_squares()
    x, y, z = system(svals, scale)
    # one source at a time: the source's mass is 1, all others 0, so the sum is that one term
    for k in range(len(svals)):
        sel = np.array([0, k + 1])
        m = np.array([0.0, 1.0])
        p = gx.ParticleSet(x[sel], y[sel], z[sel], *np.zeros((3, 2)), m)
        gx.compute_cuda_direct_accelerations(p, gx.PhysicsParams(1.0, 0.0), EXACT)
        ref = oracle.direct_targets(p.x, p.y, p.z, m, 1.0, 0.0)
        assert np.array_equal(p.accelerations, ref), svals[k]


def test_out_of_range_distances_bit_for_bit():
    """Squared distances below 2^-894 and above 2^897, zero, overflowing and infinite ones."""
    r = np.array([0.0, 2.0**-530, 3.0 * 2.0**-500, 2.0**-448, 2.0**-447, 2.0**448, 2.0**449, 1.7 * 2.0**500, 2.0**511, 2.0**513,
                  np.inf])
    x = np.concatenate([[0.0], r])
    m = np.full(len(x), 2.0**-40)
    p = gx.ParticleSet(x, x * 0.5, -x, *np.zeros((3, len(x))), m)
    gx.compute_cuda_direct_accelerations(p, gx.PhysicsParams(1.0, 0.0), EXACT)
    ref = oracle.direct_targets(p.x, p.y, p.z, m, 1.0, 0.0)
    assert np.array_equal(p.accelerations, ref, equal_nan=True)


@pytest.mark.parametrize("n", [1, 2, 15, 17, 31, 33, 63, 65, 127, 129, 255, 256, 257, 511, 1999])
def test_every_exact_variant_at_tile_edges(n):
    p = gx.ics.two_disk_encounter(n - n // 2, n // 2, 300 + n, 0.02)
    if n > 20:  # a coincident pair, skipped without softening
        p.x[9], p.y[9], p.z[9] = p.x[17], p.y[17], p.z[17]
    for eps in (0.02, 0.0):
        ref = oracle.direct_targets(p.x, p.y, p.z, p.m, 1.0, eps)
        ran = 0
        with gx.Session(n, gx.PhysicsParams(1.0, eps)) as s:
            s.set_particles(p)
            for v in range(64):
                try:
                    gx.describe_variant(EXACT, v)
                except gx.GxError:
                    continue
                s.set_config(EXACT, v, 1)
                s.compute_accelerations(EXACT)
                st = s.get_state()
                assert np.array_equal(np.stack([st["ax"], st["ay"], st["az"]], 1), ref), (v, eps)
                ran += 1
        assert ran >= 2


@pytest.mark.parametrize("n", [27000, 27001])
def test_default_variant_on_both_sides_of_the_rule(n):
    p = gx.ics.two_disk_encounter(n - n // 2, n // 2, n, 0.02)
    q = p.copy()
    gx.compute_cuda_direct_accelerations(q, gx.PhysicsParams(1.0, 0.02), EXACT)
    idx = np.concatenate([np.arange(40), np.arange(n - 40, n)])
    assert np.array_equal(q.accelerations[idx], oracle.direct_indexed(p.x, p.y, p.z, p.m, 1.0, 0.02, idx))
