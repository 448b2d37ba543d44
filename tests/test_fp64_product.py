"""The FP64 products and halved sums in integer arithmetic (csrc/k_fp64.cuh,
csrc/k_vcplane.cu), emulated with the limits of the source and compared with the
IEEE results bit by bit: ties, carries into the next power of two, both signs,
zeros, and the ends of the exponent range, where they have to decline."""
import os
import random
import re
import struct

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "libgeodecomp_gb300", "csrc")
FP64 = open(os.path.join(CSRC, "k_fp64.cuh")).read()
PLANE = open(os.path.join(CSRC, "k_vcplane.cu")).read()
LOW = 2 ** 32 - 1
M64 = 2 ** 64 - 1


def bits(x):
    return struct.unpack("<Q", struct.pack("<d", x))[0]


def value(u):
    return struct.unpack("<d", struct.pack("<Q", u))[0]


def product_bits(a, b):
    """The rounded product of the significands and the exponents' sum as the
    device forms them; the result's exponent field before the carry."""
    ua, ub = bits(a), bits(b)
    ma, mb = (ua << 11 | 1 << 63) & M64, (ub << 11 | 1 << 63) & M64
    hi, lo = ma * mb >> 64, ma * mb & M64
    big = hi >> 63
    drop = 10 + big
    odd = hi >> drop & 1
    m = (hi + (512 << big) - 1 + (odd | (lo != 0)) & M64) >> drop
    e = ((ua >> 52 & 0x7ff) + (ub >> 52 & 0x7ff) + big - 1024) & LOW
    return m, e


def mul_integer(a, b):
    span = int(re.search(r"ea != 0u && eb != 0u && e - 2u < (\d+)u", FP64).group(1))
    ua, ub = bits(a), bits(b)
    ea, eb = ua >> 52 & 0x7ff, ub >> 52 & 0x7ff
    sign = (ua ^ ub) >> 63 << 63
    m, e = product_bits(a, b)
    zero = a == 0.0 or b == 0.0
    if not (ea < 2047 and eb < 2047 and (zero or (ea and eb and (e - 2) & LOW < span))):
        return None
    return sign if zero else ((m + (e << 52)) & M64) | sign


def product(a, b):
    """a positive and normal."""
    eb_span, e_span = (int(x) for x in re.search(r"eb - 1u < (\d+)u && e - 2u < (\d+)u", PLANE).groups())
    ub = bits(b)
    m, e = product_bits(a, b)
    if b == 0.0:
        return ub
    if not (((ub >> 52 & 0x7ff) - 1) & LOW < eb_span and (e - 2) & LOW < e_span):
        return None
    return ((m + (e << 52)) & M64) | ub >> 63 << 63


def half_sum(a, b):
    alone_span, reach, span = (int(x) for x in re.search(
        r"alone \? \(ha >> 20\) - 3u < (\d+)u : \(sa \| sb\) <= (\d+)u && e0 - 3u < (\d+)u", PLANE).groups())
    ua, ub = bits(a), bits(b)
    ha, hb = ua >> 32, ub >> 32
    e0 = min(ha, hb) >> 20
    sa, sb = (ha >> 20) - e0, (hb >> 20) - e0
    if ub == 0:
        return ua - (1 << 52) if ((ha >> 20) - 3) & LOW < alone_span else None
    if not (sa | sb <= reach and (e0 - 3) & LOW < span):
        return None
    s = ((ua & (1 << 52) - 1 | 1 << 52) << sa) + ((ub & (1 << 52) - 1 | 1 << 52) << sb)
    k = s.bit_length() - 53
    assert 1 <= k <= 10
    s += (1 << k >> 1) - 1 + (s >> k & 1)
    assert s < 2 ** 64
    return (s >> k) + (e0 + k - 2 << 52)


def numbers(rng, lo, hi, signs=True):
    """Significands that make ties and carries, exponent fields lo .. hi."""
    m = rng.choice([rng.getrandbits(52), rng.getrandbits(4) << 48, rng.getrandbits(4), 2 ** 52 - 1 - rng.getrandbits(3),
                    rng.getrandbits(26) << 26, 0])
    return value((rng.getrandbits(1) if signs else 0) << 63 | rng.randint(lo, hi) << 52 | m)


@pytest.mark.parametrize("lo,hi", [(0, 2047), (1000, 1046), (0, 40), (2000, 2047), (480, 560), (1500, 1560)])
@pytest.mark.parametrize("form", [mul_integer, product])
def test_integer_product_is_the_ieee_product(form, lo, hi):
    rng = random.Random(lo)
    taken = 0
    for _ in range(30000):
        b = numbers(rng, lo, hi)
        if rng.random() < 0.02:
            b = rng.choice([0.0, -0.0, 5e-324, float("inf"), float("-inf"), float("nan")])
        if form is product:
            a = numbers(rng, 3, 2030, signs=False) if lo == 0 and hi == 2047 else numbers(rng, max(lo, 3), min(hi, 2030), False)
        else:
            a = numbers(rng, lo, hi)
        r = form(a, b)
        if r is not None:
            taken += 1
            assert r == bits(a * b), (a, b)
    assert taken > (5000 if (lo, hi) in [(0, 2047), (1000, 1046), (1500, 1560), (480, 560)] else 0)


@pytest.mark.parametrize("distance", [0, 1, 8, 9, 10, 40])
def test_integer_half_sum_is_the_ieee_one(distance):
    rng = random.Random(distance)
    taken = 0
    for _ in range(30000):
        e = rng.choice([rng.randint(0, 2047), rng.randint(0, 16), rng.randint(2020, 2047)])
        a = numbers(rng, e, e, signs=rng.random() < 0.02)
        b = numbers(rng, max(0, e - distance), min(2047, e + distance), signs=rng.random() < 0.02)
        if rng.random() < 0.05:
            b = 0.0
        r = half_sum(a, b)
        if r is not None:
            taken += 1
            assert r == bits(0.5 * (a + b)), (a, b)
    assert taken > 3000
