"""rounded.cuh: quotients and roots by fused steps have the bits of CUDA's correctly rounded ones.

The projection's chain rule, the loss, Adam and the compositing backward take their quotients and roots from
there. Operands: seeded ones over the stated ranges; the quotients that lie closest to the middle between two
floats (the only ones that a slightly wrong sum rounds the wrong way), for every odd divisor's significand; the
edges of the ranges; and, where any operand is taken, zeros, subnormals, infinities and NaN. All are compared
bit by bit (any NaN equals any other)."""
from __future__ import annotations

import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

CPP = Path(__file__).resolve().parent / "cpp"
DIVISOR, QUOTIENT, QUOTIENT2, ROOT, ADAM1, ADAM32 = range(6)
N = 1 << 22


def hard_quotients(bits=24):
    """(a, b) integers with significands of `bits` bits whose quotient is as near to the middle between two
    significands as a quotient can be: 2^e a = b m +- 1 for an odd m of bits + 1 bits."""
    lo, hi = 1 << (bits - 1), 1 << bits
    b = np.arange(lo + 1, hi, 2, dtype=np.int64)
    out = []
    for e in (bits, bits + 1):  # a >= b: the quotient's significand is from 1 to 2; a < b
        inverse = b.copy()  # of b modulo a power of two, by Newton's iteration
        for _ in range(6):
            inverse = (inverse * (2 - b * inverse)) & ((1 << e) - 1)
        for sign in (1, -1):
            m = (sign * inverse) & ((1 << e) - 1)  # b m = sign modulo 2^e
            if e == bits:
                m = m + (1 << bits)
            a = (b * m - sign) >> e
            ok = (a >= lo) & (a < hi) & (m >= (1 << bits)) & (m < (2 << bits)) & (((b * m - sign) & ((1 << e) - 1)) == 0)
            out.append((a[ok], b[ok]))
    return np.concatenate([x for x, _ in out]), np.concatenate([y for _, y in out])


def test_hard_quotients_are_next_to_the_middle():
    # Against whole numbers, at 12 bits, where all quotients can be looked at.
    a, b = hard_quotients(12)
    assert len(a) > 1000
    ints = [int(x) for x in a], [int(x) for x in b]
    distance = []
    for x, y in zip(*ints):
        e = 12 if x >= y else 13
        r = (x << e) % (2 * y)  # 2^e a = 2 b k + r: the middle is at r = b
        distance.append(abs(r - y))
    assert max(distance) == 1


@pytest.fixture(scope="module")
def lib():
    subprocess.run(["make", "-C", str(CPP), "librounding.so"], check=True, stdout=subprocess.DEVNULL)
    return C.CDLL(str(CPP / "librounding.so"))


def compare(lib, kind, a, b):
    a, b = np.ascontiguousarray(a, np.float32), np.ascontiguousarray(b, np.float32)
    fused, exact, usual = np.empty_like(a), np.empty_like(a), np.empty(len(a), np.uint8)
    p = [x.ctypes.data_as(C.c_void_p) for x in (a, b, fused, exact, usual)]
    assert lib.rounding_compare(kind, p[0], p[1], C.c_size_t(len(a)), p[2], p[3], p[4]) == 0
    same = (fused.view(np.uint32) == exact.view(np.uint32)) | (np.isnan(fused) & np.isnan(exact))
    return same, usual.astype(bool)


def powers(rng, lo, hi, n=N):
    return (np.ldexp(rng.uniform(1, 2, n), rng.integers(lo, hi, n)) * rng.choice([-1.0, 1.0], n)).astype(np.float32)


def hard(rng, aLo, aHi, bLo, bHi):
    """The hard quotients' significands at random powers of the ranges."""
    a, b = hard_quotients()
    return (np.ldexp(a.astype(np.float64), rng.integers(aLo, aHi, len(a)) - 23).astype(np.float32),
            np.ldexp(b.astype(np.float64), rng.integers(bLo, bHi, len(b)) - 23).astype(np.float32))


@pytest.mark.gpu
def test_quotients_by_a_shared_divisor(lib):
    rng = np.random.default_rng(1)
    for a, b in ((powers(rng, -83, 97), powers(rng, -30, 42)), hard(rng, -83, 97, -30, 42),
                 (np.zeros(N, np.float32) * powers(rng, 0, 1), powers(rng, -30, 42))):
        same, usual = compare(lib, DIVISOR, a, b)
        assert usual.all() and same.all(), (a[~same][:3], b[~same][:3])


@pytest.mark.gpu
def test_any_other_operands_are_known_as_such(lib):
    # Every float against every kind of divisor: where the bits are not the operator's, the caller is told.
    rng = np.random.default_rng(2)
    odd = np.array([0, 1, 2, 0x007fffff, 0x00800000, 0x00800001, 0x7f7fffff, 0x7f800000, 0x7fc00000, 0x3f800000, 0x3f7fffff],
                   np.uint32)
    odd = np.concatenate([odd, odd | 0x80000000]).view(np.float32)
    edges = np.array([np.float32(np.ldexp(m, e)) for e in (-127, -126, -83, -84, -30, -31, 42, 41, 97, 96, 126, 127)
                      for m in (1.0, 1.5, 2 - 2.0 ** -23)], np.float32)
    special = np.concatenate([odd, edges, -edges])
    x, y = (v.ravel() for v in np.meshgrid(special, special))
    any_a, any_b = (rng.integers(0, 1 << 32, N, dtype=np.uint64).astype(np.uint32).view(np.float32) for _ in range(2))
    for a, b in ((x, y), (any_a, any_b), (any_a, powers(rng, -30, 42)), (powers(rng, -83, 97), any_b),
                 (rng.choice(special, N), any_b)):
        same, usual = compare(lib, DIVISOR, a, b)
        assert (same | ~usual).all(), (a[~same & usual][:3], b[~same & usual][:3])
    # The case that a group of divisions has to be done again for: 0 over a subnormal.
    same, usual = compare(lib, DIVISOR, np.zeros(2, np.float32), np.array([1e-42, -1e-42], np.float32))
    assert not usual.any()


@pytest.mark.gpu
def test_adam_s_quotients(lib):
    rng = np.random.default_rng(3)
    for a, b in ((powers(rng, -90, 60), np.abs(powers(rng, -50, 55))), hard(rng, -90, 60, -50, 55),
                 (np.zeros(N, np.float32), np.abs(powers(rng, -50, 55)))):
        same, _ = compare(lib, QUOTIENT, a, b)
        same |= (a == 0)  # (a zero's sign does not matter there)
        assert same.all(), (a[~same][:3], b[~same][:3])
    # Every significand of a divisor.
    every = np.arange(1 << 23, 1 << 24).astype(np.float32) * np.float32(2.0 ** -23)
    for a in (np.ones(1 << 23, np.float32), powers(rng, 0, 1, 1 << 23)):
        assert compare(lib, QUOTIENT, a, every)[0].all()


@pytest.mark.gpu
@pytest.mark.parametrize("kind", [ADAM1, ADAM32])  # the smallest and the largest bias correction
def test_adam_s_range(lib, kind):
    # Step sizes times first moments over second moments of every size, their extremes together among them: where
    # the fused quotient is taken it is the operators', subnormal ones included.
    rng = np.random.default_rng(6)
    any_a, any_v = (rng.integers(0, 1 << 32, N, dtype=np.uint64).astype(np.uint32).view(np.float32) for _ in range(2))
    small, large = powers(rng, -92, -80), np.abs(powers(rng, 40, 102))
    some = 0
    for a, v in ((any_a, np.abs(any_v)), (any_a, any_v), (small, large), (powers(rng, -92, 62), np.abs(powers(rng, -102, 102))),
                 (powers(rng, 50, 62), np.abs(powers(rng, -102, -90))), (small, np.zeros(N, np.float32)),
                 (np.zeros(N, np.float32), large), (powers(rng, -60, 0), np.abs(powers(rng, -80, 10)))):
        same, usual = compare(lib, kind, a, v)
        same |= (a == 0)  # (a zero's sign does not matter there)
        assert (same | ~usual).all(), (a[~same & usual][:3], v[~same & usual][:3])
        some += usual.sum()
    assert some > 2 * N


@pytest.mark.gpu
def test_roots(lib):
    wrong = C.c_ulonglong()
    first, last = (127 - 100) << 23, (127 + 100) << 23  # every float from 2^-100 to 2^100
    assert lib.rounding_roots(first, last, C.byref(wrong)) == 0
    assert wrong.value == 0
    assert compare(lib, ROOT, np.zeros(1, np.float32), np.zeros(1, np.float32))[0].all()


@pytest.mark.gpu
def test_transmittances(lib):
    # Every divisor, one less an alpha of at most 0.99, under transmittances of every size that is stated.
    rng = np.random.default_rng(4)
    d = np.arange(int(0.01 * 2 ** 24), (1 << 24) + 1, dtype=np.int64).astype(np.float32) * np.float32(2.0 ** -24)
    for T in (np.ones(len(d), np.float32), np.abs(powers(rng, -14, 0, len(d))), np.abs(powers(rng, -90, 1, len(d)))):
        same, _ = compare(lib, QUOTIENT2, T, d)
        assert same.all(), (T[~same][:3], d[~same][:3])
    a, b = hard_quotients()
    a, b = a.astype(np.float32), b.astype(np.float32)
    b = np.where(b * np.float32(2.0 ** -24) >= 0.01, b, 2 ** 24) * np.float32(2.0 ** -24)
    same, _ = compare(lib, QUOTIENT2, a * np.float32(2.0 ** -30), b)
    assert same.all()


@pytest.mark.gpu
@pytest.mark.parametrize("culled", [False, True])
def test_gradients_of_a_gaussian_at_the_camera(culled):
    # Depths whose cubes are subnormal (below 2^-126): quotients by them are out of the fused steps' range, and
    # on the optical axis they are 0 over a subnormal, which is 0.
    from univeral_3d_reconstruction_system_b200 import api
    from univeral_3d_reconstruction_system_b200.types import GaussianModel, RasterSettings

    from helpers import make_camera
    n = 4
    m = GaussianModel.zeros(n)
    m.means[:, 2] = [1e-13, 3e-14, 2e-13, 2.0]
    m.scales[:] = np.log([1e-6, 1e-7, 2e-6, 0.1])[:, None]
    m.quats[:, 0] = 1.0
    m.opacities[:] = [-1.0, 0.0, -0.5, 0.5]
    cam, st = make_camera(33, 17, 30.0), RasterSettings(near_plane=0.0)
    w = np.random.default_rng(5).uniform(-1, 1, (17, 33, 3)).astype(np.float32)
    r = api.Rasterizer()
    r.set_tile_culling(culled)
    r.forward(m, cam, st)
    assert (r.radii() > 0).all()
    g = r.backward(m, w)
    for k in ("means", "scales", "quats", "opacities", "colors"):
        assert np.isfinite(getattr(g, k)).all(), (k, getattr(g, k))
