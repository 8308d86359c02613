"""The basis flush's shorter integer forms (csrc/flush_tc.cu), restated with Python integers on the CPU: the fixed-point
value with its shift clamped and its sign folded into the bias, digits as BF16 bit patterns, and the rounding's common
case, each equal to the plain form at random values and at the ends of its range."""
import random
import struct

import pytest

M64 = (1 << 64) - 1
DIGIT_BIAS = 0x4081020408102040


def _plain62(bits, scale):
    eb, frac = (bits >> 52) & 0x7FF, bits & ((1 << 52) - 1)
    m, r = (frac | (1 << 52) if eb else frac), 1023 + scale - max(eb, 1)
    q = (m << 10) >> r if r < 64 else 0
    return ((-q if bits >> 63 else q) + DIGIT_BIAS) & M64


def _short62(bits, scale):
    hi = bits >> 32
    eb = (hi >> 20) & 0x7FF
    m = (((hi & 0xFFFFF) | (1 << 20 if eb else 0)) << 32) | (bits & 0xFFFFFFFF)
    q = ((m << 10) & M64) >> min(1023 + scale - max(eb, 1), 63)
    return ((q ^ (M64 if bits >> 63 else 0)) + DIGIT_BIAS + (hi >> 31)) & M64


def _values():
    rng = random.Random(3)
    for eb in [0, 1, 2, 5, 1022, 1023, 1024, 2000, 2046] + [rng.randrange(2047) for _ in range(200)]:
        for frac in (0, 1, (1 << 52) - 1, rng.getrandbits(52)):
            for s in (0, 1):
                yield (s << 63) | (eb << 52) | frac


@pytest.mark.parametrize("extra", [0, 1, 5, 52, 53, 61, 62, 63, 64, 200, 2000])
def test_fixed_point(extra):
    for bits in _values():
        scale = max((bits >> 52) & 0x7FF, 1) - 1022 + extra  # |v| < 2^scale
        assert _short62(bits, scale) == _plain62(bits, scale)


def test_digits_as_bf16():
    for e in range(129):  # a digit + 64; 128 only in the top digit
        v = struct.unpack("<f", struct.pack("<I", (0x4300 | e) << 16))[0]
        assert v == 128 + e and v - 192 == e - 64


def _join(T, k):
    """T 2^k, half up on the magnitude's 53 leading bits, by exact integers."""
    a = abs(T)
    if a == 0:
        return 0
    z = 64 - a.bit_length()
    w = a << z
    return ((63 - z + k + 1022) << 52) + (w >> 11) + ((w >> 10) & 1) | (1 << 63 if T < 0 else 0)


def _join_short(T, k):
    a, ah = abs(T), abs(T) >> 32
    z = 32 - ah.bit_length()
    e = 1085 - z + k
    if a != 0 if ah == 0 else not 0 <= e <= 2044:
        return None  # the out-of-line form
    w = (a << z) & M64
    mant = (w >> 11) + (((w & 0xFFFFFFFF) >> 10) & 1)
    hi = (mant >> 32) + (e << 20) if ah else 0
    return ((hi | (1 << 31 if T < 0 else 0)) << 32) | (mant & 0xFFFFFFFF)


@pytest.mark.parametrize("k", [-1090, -700, -56, 0, 11, 900, 960])
def test_rounding(k):
    rng = random.Random(k)
    cases = [0, 1 << 32, (1 << 63) - 1, (1 << 62) + (1 << 8), (1 << 53) - 1, (1 << 54) - 1, (1 << 33) + 1]
    cases += [rng.getrandbits(rng.randrange(1, 64)) for _ in range(3000)]
    short = 0
    for a in cases:
        for T in (a, -a):
            got = _join_short(T, k)
            if got is not None:
                short += 1
                assert got == _join(T, k)
            else:
                assert 0 < abs(T) < 1 << 32 or not 0 <= abs(T).bit_length() + k + 1021 <= 2044
    assert short > 1000 or k < -1000
