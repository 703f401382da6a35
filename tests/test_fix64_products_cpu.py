"""rn_product and Factor (fix64.cuh), restated in exact Python integers: FP64
products rounded to nearest even on the integer pipes, bit for bit those of the
FP64 multiplier (CPU).  The phases' bits rest on it.

Also the sampled maximum that the header states for the cosine's error, with the
phase where it was found.
"""
import os
import random
import re
import struct

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = open(os.path.join(HERE, "..", "gstools-core_gb300", "csrc", "fix64.cuh")).read()
M32, M64 = (1 << 32) - 1, (1 << 64) - 1


def bits(x):
    return struct.unpack("<Q", struct.pack("<d", x))[0]


def double(b):
    return struct.unpack("<d", struct.pack("<Q", b))[0]


def factor(x):
    """(m1, m0, e), as factor_of."""
    hi, lo = bits(x) >> 32, bits(x) & M32
    if x == 0.0:
        return 0x80000000, 0, (1023 - 450) << 20
    return ((hi << 11) | (lo >> 21)) & M32 | 0x80000000, (lo << 11) & M32, hi & 0xFFF00000


def value(f):
    m1, m0, e = f
    return double((e | ((m1 << 1) & M32) >> 12) << 32 | ((m1 << 32 | m0) >> 11) & M32)


def in_range(x):
    e = (bits(x) >> 52 & 0x7FF) - 1023
    return x == 0.0 or -200 <= e <= 200


def funnel_l(lo, hi, n):
    return (hi << n | lo >> (32 - n)) & M32 if n else hi


def rn_product(x, y):
    (x1, x0, xe), (y1, y0, ye) = x, y
    t = x0 * y0
    u = x1 * y0 + (t >> 32)
    v = x0 * y1 + (u & M32)
    w = x1 * y1 + (u >> 32) + (v >> 32)
    assert max(u, v, w) <= M64
    h, l, m = w >> 32, w & M32, v & M32
    up = (h >> 31) ^ 1
    h2, l2 = funnel_l(l, h, up), funnel_l(m, l, up)
    rest = min((m << up) & M32 | t & M32, 1)
    below = (l2 & 0x7FF) | rest
    lo = (h2 << 32 | l2) >> 11 & M32
    inc = (below + 0x3FF + (lo & 1)) >> 11
    e = (xe + ye - (1023 << 20) - (up << 20)) & M32
    r = ((((h2 >> 11) + e) & M64) << 32 & M64 | lo) + inc & M64
    return double(r)


def test_the_restatement_is_of_this_source():
    body = SRC.split("rn_product(const Factor &x, const Factor &y) {")[1].split("\n}")[0]
    for line in ("const uint64_t t = static_cast<uint64_t>(x.m0) * y.m0;",
                 "static_cast<uint64_t>(x.m1) * y.m0 + (t >> 32);",
                 "static_cast<uint64_t>(x.m0) * y.m1 + static_cast<uint32_t>(u);",
                 "static_cast<uint64_t>(x.m1) * y.m1 + (u >> 32) + (v >> 32);",
                 "min((m << up) | static_cast<uint32_t>(t), 1u);",
                 "(below + 0x3ffu + (lo & 1u)) >> 11;",
                 "x.e + y.e - (static_cast<uint32_t>(1023) << 20) - (up << 20);"):
        assert line in body, line
    assert re.search(r"e >= -200 && e <= 200", SRC)


def check(x, y):
    assert in_range(x) and in_range(y)
    for a in (x, -x):
        for b in (y, -y):
            assert bits(rn_product(factor(a), factor(b))) == bits(a * b), (a, b)


def test_random_products():
    rng = random.Random(1)
    for _ in range(40_000):
        check(rng.uniform(1.0, 2.0) * 2.0 ** rng.randint(-200, 200), rng.uniform(1.0, 2.0) * 2.0 ** rng.randint(-200, 200))


def test_exact_ties():
    """Products of 54 significant bits: halfway between two doubles, to either neighbour."""
    rng = random.Random(2)
    found = {0: 0, 1: 0}
    while min(found.values()) < 2000:
        a, b = rng.getrandbits(27) | 1 | 1 << 26, rng.getrandbits(27) | 1 | 1 << 26
        p = a * b
        if p.bit_length() != 54:
            continue
        found[p >> 1 & 1] += 1
        check(a * 2.0 ** rng.randint(-100, 100), b * 2.0 ** rng.randint(-100, 100))
    # one bit more or less than a tie
    for _ in range(2000):
        a, b = rng.getrandbits(53) | 1 << 52 | 1, rng.getrandbits(3) | 1
        check(float(a), float(b))


def test_carries_into_the_exponent():
    """Products that round up to a power of two, and the largest mantissas."""
    rng = random.Random(3)
    top = 2.0 - 2.0 ** -52
    for x, y in ((top, top), (top, 1.0), (1.0, 1.0), (top, 1.0 + 2.0 ** -52), (1.0 + 2.0 ** -52, 1.0 + 2.0 ** -52)):
        check(x, y)
        check(x * 2.0 ** 200, y * 2.0 ** -200)
    up = 0
    for _ in range(200_000):
        x = rng.uniform(1.0, 2.0)
        y = 2.0 / x                               # the product is next to 2
        if x * y == 2.0:
            up += 1
            check(x, y)
        if up >= 3000:
            break
    assert up >= 3000


def test_zero_factors_and_values():
    """A zero stands for 2^-450: its products are far below any phase's last bit."""
    for y in (1.0, -3.5, 2.0 ** 200, 2.0 ** -200, 0.0):
        assert abs(rn_product(factor(0.0), factor(y))) <= 2.0 ** -249
        assert abs(rn_product(factor(y), factor(-0.0))) <= 2.0 ** -249
    rng = random.Random(4)
    for _ in range(5000):
        x = rng.choice((1, -1)) * rng.uniform(1.0, 2.0) * 2.0 ** rng.randint(-200, 200)
        assert value(factor(x)) == x
    assert value(factor(0.0)) == 2.0 ** -450


def test_sampled_maximum_of_the_cosine():
    mp = pytest.importorskip("mpmath")
    from test_fix64_cpu import OFFSET, cos_fixed
    stated = float(re.search(r"RMS, ([0-9.]+)e-16 the\n//\s+largest of", SRC).group(1)) * 1e-16
    rng = random.Random(5)
    near = [((q << 62) + rng.randint(-(1 << 55), 1 << 55)) % (1 << 64) for q in range(4) for _ in range(300)]
    with mp.workprec(300):
        def error(th):
            return abs(mp.mpf(cos_fixed(th)) / mp.mpf(2) ** 62
                       - mp.cos(2 * mp.pi * mp.mpf(th - OFFSET) / mp.mpf(2) ** 64))
        worst = error(0xC002A71564FDAD2A)
        assert abs(worst - stated) <= 0.05e-16
        assert max(error(th) for th in near) <= 9e-16      # the derived bound
