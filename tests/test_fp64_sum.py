"""sum4 (csrc/k_fp64.cuh), the rounded sum of four doubles in integer
arithmetic, emulated with the constants of the source and compared with the
IEEE sum bit by bit: exponents up to and beyond the accepted distance, ties,
carries into the next power of two, both signs, and a dropped zero."""
import os
import random
import re
import struct

import pytest

SRC = open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "libgeodecomp_gb300", "csrc",
                        "k_fp64.cuh")).read()
REACH = int(re.search(r"#define LGD_FP64_SUM_REACH (\d+)", SRC).group(1))
SPAN = int(re.search(r"reach <= LGD_FP64_SUM_REACH && e0 - 1u < (\d+)u", SRC).group(1))
LOW = 2 ** 32 - 1


def bits(x):
    return struct.unpack("<Q", struct.pack("<d", x))[0]


def value(u):
    return struct.unpack("<d", struct.pack("<Q", u))[0]


def integer_form(a, drop):
    """The device's integer sum, or None where it adds in FP64."""
    u = [bits(x) for x in a]
    sign = u[0] >> 63 << 31
    h = [(w >> 32) ^ sign for w in u]
    if drop:
        h[3] = h[0]
    e0 = ((min(h) >> 20) - 1) & LOW
    shift = [((w >> 20) - e0) & LOW for w in h]
    if shift[0] | shift[1] | shift[2] | shift[3] > REACH or (e0 - 1) & LOW >= SPAN:
        return None
    v = [((w & 0xFFFFF | 0x100000) << 32 | x & LOW) << n for w, x, n in zip(h, u, shift)]
    if drop:
        v[3] = 0
    s = v[0]
    for x in v[1:]:
        s += x
        k = s.bit_length() - 53
        assert 1 <= k <= 10
        s += (1 << k >> 1) - 1 + (s >> k & 1)
        s &= ~((1 << k) - 1)
        assert s < 2 ** 63
    return (s >> k) + ((e0 + k - 1) << 52) | sign << 32


@pytest.mark.parametrize("reach", [0, 1, 6, 7])
@pytest.mark.parametrize("drop", [False, True])
def test_integer_sum_is_the_ieee_sum(reach, drop):
    rng = random.Random(reach)
    seen = 0
    for _ in range(30000):
        e = rng.randrange(0, 2048)
        sign = rng.getrandbits(1)

        def one():
            m = rng.choice([rng.getrandbits(52), rng.getrandbits(4) << 48, rng.getrandbits(4),
                            2 ** 52 - 1 - rng.getrandbits(3), rng.getrandbits(26) << 26])
            s = sign if rng.random() < 0.98 else 1 - sign
            return value(s << 63 | min(2047, e + rng.randint(0, reach)) << 52 | m)

        a = [one() for _ in range(4)]
        if drop:
            a[3] = rng.choice([0.0, -0.0])
        r = integer_form(a, drop)
        if r is not None:
            seen += 1
            assert r == bits(((a[0] + a[1]) + a[2]) + a[3]), a
    assert seen > 15000
