"""turn_fraction_far (fix64.cuh), restated in exact Python integers from the
header's constants: phases below 2^44 as fractions of a turn (CPU).

Bound: the product's dropped words are below two units of its bit 64, which the
shift of 22 bits or more puts below 2^-21 units of 2^-64 turn; the shift drops
less than one unit, and a negative phase is the one's complement: 2 units.
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
PLAIN = open(os.path.join(HERE, "..", "gstools-core_gb300", "csrc", "plain.cu")).read()
CH, CL = (int(v, 16) for v in re.search(r"ch = 0x(\w+)ull, cl = 0x(\w+)ull", SRC).groups())
M64 = (1 << 64) - 1


def far(ph):
    bits = struct.unpack("<Q", struct.pack("<d", ph))[0]
    m = (bits << 11) & M64 | 1 << 63
    lo = m * CH & M64
    low = (lo + (m * CL >> 64)) & M64
    high = (m * CH >> 64) + (1 if low < lo else 0)
    assert high <= M64
    s = 1088 - (bits >> 52 & 0x7FF)
    assert s >= 22
    f = (high << (64 - s) | low >> s) & M64 if s < 64 else high >> (s - 64) if s < 128 else 0
    return f ^ (M64 if bits >> 63 else 0)


def _error(ph):
    """In units of 2^-64 turn, the short way round."""
    with mp.workprec(400):
        want = mpf(ph) / (2 * mp.pi)
        d = mpf(far(ph)) / mpf(2) ** 64 - want
        return abs(d - mp.nint(d)) * mpf(2) ** 64


def test_constants_and_range():
    with mp.workprec(400):
        assert CH << 64 | CL == int(mp.floor(2 / mp.pi * mpf(2) ** 128))
    limit = float(re.search(r"kFarPhase = ([0-9.e]+)f", PLAIN).group(1))
    assert limit * (1 + 1e-6) < 2.0 ** 44


def test_every_exponent():
    rng = random.Random(1)
    for e in list(range(-80, 44)) + [-1000, -300, -129]:
        for _ in range(60):
            ph = rng.uniform(1.0, 2.0) * 2.0 ** e
            assert _error(ph) <= 2 and _error(-ph) <= 2
        for ph in (2.0 ** e, 2.0 ** e * (2.0 - 2.0 ** -52)):
            assert _error(ph) <= 2 and _error(-ph) <= 2


def test_zero_subnormal_and_whole_turns():
    for ph in (0.0, -0.0, 5e-324, -2.0 ** -1040):
        assert _error(ph) <= 2
    for turns in (1, 7, 683565276, 1591549430918):     # FP64 values next to whole turns, up to 1e13
        with mp.workprec(400):
            ph = float(2 * mp.pi * turns)
        assert _error(ph) <= 2 and _error(-ph) <= 2
