"""gelu_pair (csrc/tc_common.cuh), restated with the constants of the source: the
fits' errors in FP64 and the results' in FP32 (reciprocal and exponential
correctly rounded, small results flushed) against erfc and exp, each within what
the comment beside it states."""
import math
import os
import re

import numpy as np

SRC = open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "libgeodecomp_gb300", "csrc",
                        "tc_common.cuh")).read()
F = np.float32


def constants(name):
    m = re.search(r"constexpr float %s(?:\[\d+\])? = \{?([^;]*?)\}?;" % name, SRC, re.S).group(1)
    return [float(F(x.strip().rstrip("f"))) for x in m.split(",")]


(P,), C, Q = constants("P"), constants("C"), constants("Q")
erfc = np.vectorize(math.erfc)


def stated(pattern):
    return float(re.search(pattern, re.sub(r"\s*\n//\s*", " ", SRC)).group(1))


def fma(a, b, c):
    return F(np.float64(a) * np.float64(b) + np.float64(c))


def flushed(x):
    return np.where(np.abs(x) < 2.0 ** -126, F(0), F(x))


def gelu_pair(z):
    s = F(z * z)
    t = F(1 / np.float64(fma(np.abs(z), F(P), F(1))))
    e = flushed(np.exp2(np.float64(F(s * F(-0.72134752)))))
    p, r = np.full_like(z, C[6]), np.full_like(z, Q[4])
    for i in range(5, -1, -1):
        p = fma(p, t, F(C[i]))
    for i in range(3, -1, -1):
        r = fma(r, s, F(Q[i]))
    r, te = fma(r, z, F(0.5)), F(t * e)
    phi = np.where(s < 1, r, np.where(z >= 0, fma(-p, te, F(1)), F(p * te)))
    return F(z * phi), fma(F(e * F(0.39894228)), z, phi), phi


def test_fits():
    z = np.linspace(0, 1, 40001)
    err = np.abs(0.5 + z * np.polyval(Q[::-1], z * z) - 0.5 * erfc(-z / math.sqrt(2)))
    assert err.max() < stated(r"Q of degree 4 \((?:error of the fit below|largest error) ([\d.e-]+)\)")
    z = np.linspace(1, 14, 40001)
    t = 1 / (1 + P * z)
    err = np.abs(np.exp(-z * z / 2) * t * np.polyval(C[::-1], t) / (0.5 * erfc(z / math.sqrt(2))) - 1)
    assert err.max() < stated(r"\(relative error (?:of the fit below )?([\d.e-]+) up to z = 14")


def test_fp32_results():
    z = F(np.linspace(-16, 16, 200001))
    h, g, phi = gelu_pair(z)
    x = np.float64(z)
    exact = 0.5 * erfc(-x / math.sqrt(2))
    assert np.abs(h - x * exact).max() < stated(r"GELU is within ([\d.e-]+) \(")
    assert np.abs(g - exact - x * np.exp(-x * x / 2) / math.sqrt(2 * math.pi)).max() < stated(r"GELU' within ([\d.e-]+);")
    rel = np.abs(phi / exact - 1)
    assert rel[x >= -4].max() < stated(r"lower tail is within ([\d.e-]+) to z = -4")
    assert rel[x >= -13.2].max() < stated(r"and ([\d.e-]+) to z = -13.2")
    assert not phi[x < -13.3].any()
