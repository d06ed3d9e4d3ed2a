"""The rounding of an update's integer sum in integer instructions (emu::round_scaled, ttg_gb300/csrc/emu_f64.cuh),
restated step by step in 32-bit words, against the exact product of the rounded sum and 2^sE: every bit length of the sum
that it takes, ties and carries, both signs, and the scales at the ends of its range; shorter sums are left to the
conversion."""
import math
import random
import struct

import pytest

M32 = 0xFFFFFFFF


def _clz(x):
    return 32 - x.bit_length()


def _funnel_l(lo, hi, s):
    s &= 31
    return (((hi << 32 | lo) << s) >> 32) & M32


def _funnel_r(lo, hi, s):
    return ((hi << 32 | lo) >> (s & 31)) & M32


def round_scaled(X, sE):
    a = abs(X)
    ah, al = a >> 32, a & M32
    wide = ah == 0 or (sE + 1022) & M32 > 1980
    z = _clz(ah)
    mh, ml = _funnel_l(al, ah, z), (al << (z & 31)) & M32
    lo = _funnel_r(ml, mh, 11)
    up = ((ml & 0x7FF) + 0x3FF + (lo & 1)) >> 11
    m = ((mh >> 11) << 32 | lo) + up
    hi = (((m >> 32) + (((1085 - z + sE) << 20) & M32)) & M32) | (0x80000000 if X < 0 else 0)
    return struct.unpack("<d", struct.pack("<II", m & M32, hi))[0], wide


def _sums():
    rng = random.Random(1)
    for bits in range(33, 64):
        yield 1 << (bits - 1)
        yield (1 << bits) - 1
        for _ in range(40):
            a = rng.getrandbits(bits) | 1 << (bits - 1)
            yield a
            if bits > 54:  # ties, and what rounds up into the next power of two
                low = bits - 53
                yield a >> low << low | 1 << (low - 1)
                yield (1 << bits) - 1 - rng.getrandbits(low)


@pytest.mark.parametrize("sE", [-1022, -1021, -700, -62, -1, 0, 1, 500, 957, 958])
def test_round_scaled_is_the_rounded_sum_times_the_scale(sE):
    for a in _sums():
        for X in {a, -a}:
            d, wide = round_scaled(X, sE)
            assert not wide
            assert d == math.ldexp(float(X), sE) and math.copysign(1, d) == (-1 if X < 0 else 1)


@pytest.mark.parametrize("sE", [-1023, 959, 100000, -8000])
def test_scales_outside_are_wide(sE):
    assert round_scaled(1 << 40, sE)[1]


def test_short_sums_are_wide():
    assert all(round_scaled(X, 0)[1] for X in (0, 1, -1, (1 << 32) - 1)) and not round_scaled(1 << 32, 0)[1]
