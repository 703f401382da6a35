"""The 64-bit fixed-point cosine of the FP64 kernels (fix64.cuh), restated in
exact Python integers from the header's constants (CPU).

Checked against 300-bit arithmetic: the turn fraction of FP64 phases within
2^-60 turn, at every exponent it accepts, zero and subnormal phases included;
the cosine within 9e-16 everywhere: 1.8e-16 from the sixth-order fit and at
most two units of 2^-46 of a table step (0.0245 rad), 7e-16, from the
truncated products of the sine's cubic term; the factor tables' finer cosine
and sine within 1e-17.  Every intermediate stays inside
the word the kernel holds it in.
"""
import os
import random
import re
import struct

import pytest

mpmath = pytest.importorskip("mpmath")
from mpmath import mp, mpf  # noqa: E402

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = open(os.path.join(HERE, "..", "gstools-core_gb300", "csrc", "fix64.cuh")).read()
M32, M64 = (1 << 32) - 1, (1 << 64) - 1


def _const(name):
    v = re.search(r"constexpr uint(?:32|64)_t " + name + r" = (0x[0-9a-f]+|\d+)u", SRC).group(1)
    return int(v, 0)


QUARTER = [int(v, 16) for v in re.findall(r"0x([0-9a-f]{16})ull", SRC.split("kQuarterCos[65]")[1].split("};")[0])]
STEP, A1, A2 = _const("kStep69"), _const("kVersine75"), _const("kVersineTwo")
S3, S5 = _const("kSineThree"), _const("kSineFive")
TWO_OVER_PI = [int(v, 16) for v in re.search(r"c2 = 0x(\w+)u, c1 = 0x(\w+)u, c0 = 0x(\w+)u", SRC).groups()]
OFFSET = (1 << 55) - (1 << 9)


@pytest.fixture(autouse=True)
def _precision():
    with mp.workprec(300):
        yield


def s32(x):
    assert 0 <= x <= M32
    return x - (1 << 32) if x >> 31 else x


def mulhi(a, b):
    assert -2**31 <= a < 2**31 and -2**31 <= b < 2**31
    return (a * b) >> 32


def umulhi(a, b):
    assert 0 <= a <= M32 and 0 <= b <= M32
    return (a * b) >> 32


def i64(x):
    assert -2**63 <= x < 2**63
    return x


def quarter_cos(a):
    a &= 255
    b = a & 127
    v = QUARTER[b if b <= 64 else 128 - b]
    return -v if (a + 64) & 128 else v


def table_entry(a):
    c, s = quarter_cos(a), quarter_cos(a - 64)
    ss, cc = (abs(s) * STEP >> 64) << 1, (abs(c) * A1 >> 64) >> 5
    return c, -ss if s < 0 else ss, -cc if c < 0 else cc


def turn_fraction(ph):
    bits = struct.unpack("<Q", struct.pack("<d", ph))[0]
    hi, lo = bits >> 32, bits & M32
    c2, c1, c0 = TWO_OVER_PI
    m1, m0 = ((hi << 11) | (lo >> 21)) & M32 | 0x80000000, (lo << 11) & M32
    t0 = ((hi >> 20) & 0x7FF) - 992
    down, t = max(-t0, 0), max(t0, 0)
    m0 = ((m1 << 32 | m0) >> min(down, 32)) & M32
    m1 = m1 >> down if down < 32 else 0
    w = umulhi(m1, c0) + umulhi(m0, c1) + m0 * c2 + m1 * c1
    assert w <= M64
    p2 = w & M32
    w = m1 * c2 + (w >> 32)
    assert w <= M64
    p3, p4 = w & M32, w >> 32
    a, b, c = (p4, p3, p2) if t & 32 else (0, p4, p3)
    t &= 31
    fh, fl = ((a << 32 | b) << t) >> 32 & M32, ((b << 32 | c) << t) >> 32 & M32
    if hi >> 31:
        fh, fl = fh ^ M32, fl ^ M32
    return fh << 32 | fl


def cos_fixed(theta):
    h, l = theta >> 32, theta & M32
    c, es, ec = table_entry(h >> 24)
    r1 = s32(((h << 8 | l >> 24) & M32) ^ 0x80000000)
    r0 = (l << 7) & 0x7FFFFFFF
    sq = i64(r1 * r1 + 4 + (mulhi(r1, r0) << 2))
    assert sq >= 0
    q = ((sq & M64) >> 31) & M32
    assert sq >> 31 <= M32
    a2 = umulhi(umulhi(q, q), A2)
    v = i64(sq - (s32(a2) << 17))
    s3 = umulhi(q, S3 - umulhi(q, S5))
    s = i64(((r1 << 32) | ((l << 8) & M32)) - (mulhi(r1, s32(s3)) << 18))
    vh, v0, sh, s0 = v >> 32, (v & M32) >> 1, s >> 32, (s & M32) >> 1
    eh, e0, fh, f0 = es >> 32, (es & M32) >> 1, ec >> 32, (ec & M32) >> 1
    low = mulhi(fh, v0) + mulhi(f0, vh) + mulhi(eh, s0)
    assert -2**31 <= low < 2**31
    p = i64(eh * sh + fh * vh + (low << 1) + (mulhi(e0, sh) << 1))
    return c - (p >> 6)


FINE = [None] + [_const("kFine%d" % i) for i in range(1, 6)]


def mul64hi(a, b):
    return i64(a) * i64(b) >> 64


def umul64hi(a, b):
    assert 0 <= a <= M64 and 0 <= b <= M64
    return a * b >> 64


def cis_fine(theta):
    a = theta >> 56
    c, s = quarter_cos(a), quarter_cos(a + 192)
    rho = ((theta << 8) & M64) - 2**63
    q = mul64hi(rho, rho) << 1
    lv = umul64hi(q, FINE[2] - umul64hi(q, FINE[3]))
    ls = umul64hi(q, FINE[4] - umul64hi(q, FINE[5]))
    ver = umul64hi(q - (umul64hi(q, lv) >> 13), FINE[1])
    sn = mul64hi(rho - (mul64hi(rho, ls) >> 12), STEP >> 1)
    return (c - (((mul64hi(c, ver) >> 8) + mul64hi(s, sn) + 8) >> 4),
            s - (((mul64hi(s, ver) >> 8) - mul64hi(c, sn) + 8) >> 4))


def _turn_error(ph):
    exact = mpf(ph) / (2 * mp.pi)
    d = mpf(turn_fraction(ph)) / mpf(2) ** 64 - exact
    return abs(d - mp.nint(d))


def test_constants():
    assert len(QUARTER) == 65
    for a, v in enumerate(QUARTER):
        assert v == int(mp.nint(mp.cos(2 * mp.pi * a / 256) * mpf(2) ** 62))
    assert TWO_OVER_PI[0] << 64 | TWO_OVER_PI[1] << 32 | TWO_OVER_PI[2] == int(mp.floor(mpf(2) ** 97 / mp.pi))
    assert STEP == int(mp.nint(2 * mp.pi / 256 * mpf(2) ** 69))


def test_turn_fraction():
    rng = random.Random(5)
    for e in range(-60, 32):
        for _ in range(12):
            ph = rng.choice((1, -1)) * rng.uniform(1.0, 2.0) * 2.0 ** e
            assert _turn_error(ph) <= mpf(2) ** -60, ph
    for ph in (0.0, -0.0, 5e-324, -1e-310, 1e-300, 2.0 ** -31, 2.0 ** -32, 2.0 ** -63, 2.0 ** -64,
               float(mpf(2) ** 32 * (1 - mpf(2) ** -53)), 1.0, 3.0, 1e9 + 1 / 3):
        assert _turn_error(ph) <= mpf(2) ** -60, ph


def test_cosine():
    rng = random.Random(6)
    thetas = [rng.getrandbits(64) for _ in range(4000)]
    # both ends and the middle of every table cell
    thetas += [((a << 56) + off) & M64 for a in range(256) for off in (0, 1, -1, 1 << 55, (1 << 55) - 1, (1 << 32) - 1)]
    square = 0.0
    for th in thetas:
        err = abs(mpf(cos_fixed(th)) / mpf(2) ** 62 - mp.cos(2 * mp.pi * mpf(th - OFFSET) / mpf(2) ** 64))
        assert err <= 9e-16, hex(th)
        square += float(err) ** 2
    assert (square / len(thetas)) ** 0.5 <= 2e-16


def test_fine_cosine_and_sine():
    """8.4e-18 of the sine's next term, and a few units of 2^-62 of rounding."""
    rng = random.Random(7)
    thetas = [rng.getrandbits(64) for _ in range(2000)]
    thetas += [((a << 56) + off) & M64 for a in range(256) for off in (0, 1, -1, 1 << 55)]
    for th in thetas:
        angle = 2 * mp.pi * mpf(th - (1 << 55)) / mpf(2) ** 64
        c, s = cis_fine(th)
        assert abs(mpf(c) / mpf(2) ** 62 - mp.cos(angle)) <= 1e-17, hex(th)
        assert abs(mpf(s) / mpf(2) ** 62 - mp.sin(angle)) <= 1e-17, hex(th)
