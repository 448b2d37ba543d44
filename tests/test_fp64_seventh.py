"""mul_seventh (csrc/k_fp64.cuh), the product with fl(1/7) in integer
arithmetic, emulated with the constants of the source and compared with the
IEEE product bit by bit: random bit patterns, random significands, and the
neighbourhood of the four significands whose product is a tie (which the
device sends to the FP64 multiplication, as it does everything outside the
exponent range)."""
import os
import random
import re
import struct

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "libgeodecomp_gb300", "csrc")
C7 = int(re.search(r"#define LGD_FIX_C7 (\d+)ull", open(os.path.join(CSRC, "k_common.cuh")).read()).group(1))
SRC = open(os.path.join(CSRC, "k_fp64.cuh")).read()
SHIFT = int(re.search(r"#define LGD_FP64_C7_SHIFT (\d+)", SRC).group(1))
LOW, SPAN, MASK = (int(v, 0) for v in re.search(
    r"e - (\d+)u < (\d+)u && \(u & (0x[0-9a-f]+)ull\) != 0", SRC).groups())


def bits(x):
    return struct.unpack("<Q", struct.pack("<d", x))[0]


def value(u):
    return struct.unpack("<d", struct.pack("<Q", u))[0]


def integer_form(u):
    """The device's integer product, or None where it multiplies in FP64."""
    e = (u >> 52) & 0x7FF
    if not (LOW <= e < LOW + SPAN) or not u & MASK:
        return None
    hi = ((((u << 11) & (2 ** 64 - 1)) | 1 << 63) * (C7 << SHIFT)) >> 64
    big = hi >> 63
    m = hi + (512 << big)
    assert m < 2 ** 64
    return ((m >> (10 + big)) + ((e - 4 + big) << 52)) | (u & 1 << 63)


def patterns(kind, rng):
    e = rng.randrange(0, 2048) << 52
    if kind == "any":
        return rng.getrandbits(64)
    if kind == "unit":
        return 1022 << 52 | rng.getrandbits(52)
    if kind == "sparse":
        return e | rng.getrandbits(12) << 40 | rng.choice([0, 1, 2, (1 << 40) - 1])
    return e | (rng.choice([0, 1, 2, 3]) * 2 ** 50 + rng.randrange(-4, 5)) & (2 ** 52 - 1)


@pytest.mark.parametrize("kind", ["any", "unit", "sparse", "ties"])
def test_integer_product_is_the_ieee_product(kind):
    rng = random.Random(7)
    seen = 0
    for _ in range(60000):
        u = patterns(kind, rng)
        r = integer_form(u)
        if r is not None:
            seen += 1
            assert r == bits(value(u) * (1.0 / 7.0)), hex(u)
    assert seen > 20000
