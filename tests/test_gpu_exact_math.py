"""The passes' block forms of division and square root return the IEEE values:
on random operands in and beyond their range, on special values, and on the
hardest operands there are (quotients and roots nearest to a rounding
boundary, built with integer arithmetic)."""
import ctypes as C
import math

import numpy as np
import pytest

import physics_engine_rs as pe

pytestmark = pytest.mark.gpu


def mismatches(num, den):
    f = pe.load_library().pe_fluid_probe_exact_math
    f.restype, f.argtypes = C.c_int, [C.c_int32, C.c_uint64, C.c_void_p, C.c_void_p, C.c_void_p]
    num, den = np.ascontiguousarray(num, np.float64), np.ascontiguousarray(den, np.float64)
    out = np.zeros(4, np.uint64)
    assert f(-1, num.size, num.ctypes.data, den.ctypes.data, out.ctypes.data) == 0
    return [int(v) for v in out]


def random_operands(rng, n, exp):
    """Doubles with uniform significands and exponents in [-exp, exp], some significands near 1 or 2."""
    m = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    near = rng.integers(0, 64, n, dtype=np.uint64)
    kind = rng.integers(0, 8, n)
    m = np.where(kind == 0, near, np.where(kind == 1, (1 << 52) - 1 - near, m)).astype(np.uint64)
    e = rng.integers(1023 - exp, 1024 + exp, n).astype(np.uint64)
    return (m | (e << np.uint64(52))).view(np.float64)


@pytest.mark.parametrize("exp", [20, 127, 140, 1000])
def test_random_operands(exp):
    rng = np.random.default_rng(exp)
    n = 1 << 23
    num = random_operands(rng, n, exp) * rng.choice((-1.0, 1.0), n)
    num[rng.integers(0, n, 1000)] = 0.0
    bad = mismatches(num, random_operands(rng, n, exp))
    assert bad[:3] == [0, 0, 0]
    assert bad[3] > (0.99 * n if exp <= 20 else 0)


def test_special_values():
    v = np.array([0.0, -0.0, 1.0, -1.0, np.inf, -np.inf, np.nan, 5e-324, 2.2e-308, 1.7e308, 2.0**-128, 2.0**128,
                  np.nextafter(2.0**-128, 0), np.nextafter(2.0**128, 0), np.nextafter(2.0, 0), 1e-30, 1e-60])
    a, b = np.meshgrid(v, v)
    assert mismatches(a.ravel(), b.ravel())[:3] == [0, 0, 0]


def test_hardest_quotients():
    """n 2^53 - M d = c for small odd c and odd M: n / d lies c / d from the midpoint M / 2^53."""
    rng = np.random.default_rng(7)
    num, den = [], []
    for k in range(20000):
        d = int(rng.integers(1 << 52, 1 << 53)) | 1
        if k % 3 == 0:
            d = (1 << 53) - 1 - 2 * int(rng.integers(0, 4096))
        inv = pow(d, -1, 1 << 53)
        for c in (1, -1, 3, -3):
            m = (-c * inv) % (1 << 53) | (1 << 53)
            p = m * d + c
            n = p >> 53
            if p & ((1 << 53) - 1) == 0 and n < (1 << 54) and (n < (1 << 53) or n % 2 == 0):
                num.append(float(n))
                den.append(float(d))
    assert len(num) > 20000
    bad = mismatches(num, den)
    assert bad[0] == 0 and bad[3] > 0.99 * len(num)


def test_hardest_roots():
    """M^2 = a 2^k + c for small c and 54-bit M: sqrt(a) lies c / (2 M) from a midpoint."""
    rad = []
    for k in (53, 54, 55, 56):
        for c in range(-4095, 4096):
            if c % 8 != 1:
                continue
            for x in (1, 3, 5, 7):
                for j in range(3, k):
                    if (x * x - c) >> j & 1:
                        x += 1 << (j - 1)
                if (x * x - c) % (1 << k):
                    continue
                x %= 1 << (k - 1)
                for t in range((1 << 54 >> (k - 1)) + 1):
                    m = x + (t << (k - 1))
                    a = (m * m - c) >> k
                    if 1 << 53 <= m < 1 << 54 and (m * m - c) % (1 << k) == 0 and a < 1 << 53:
                        rad += [math.ldexp(a, k % 2), math.ldexp(a, k % 2 - 60)]
    assert len(rad) > 1000
    assert mismatches(np.ones(len(rad)), rad)[:3] == [0, 0, 0]
