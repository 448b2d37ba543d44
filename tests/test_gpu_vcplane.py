"""The one-cell-per-thread var-coef kernel (csrc/k_vcplane.cu): FP64 bit for bit
against the oracle on tori and against the kernel of variant 1 for every set of
wrapping axes and edge values, with coefficients and fields at the ends of the
exponent range; FP32 grids of ragged rows against variant 1."""
import numpy as np
import pytest

import oracle
from libgeodecomp_gb300 import lgd

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 127), (3, 2, 1), (2, 16, 8), (17, 1, 129), (9, 33, 31), (40, 20, 66)]


def run(cell, u, k, steps, variant, periodic, edge=(0.0, 0.0, 0.0, 0.0)):
    with lgd.Grid(cell, u.shape, periodic=periodic, edge=edge) as g:
        g.set_variant(variant)
        g.upload(0, u)
        g.upload(1, k)
        g.step(steps)
        return g.download(0)


def fields(shape, seed):
    rng = np.random.default_rng(seed)
    return rng.random(shape), 0.02 + 0.13 * rng.random(shape)


@pytest.mark.parametrize("shape", SHAPES)
def test_fp64_torus_matches_oracle(shape):
    u, k = fields(shape, 1)
    np.testing.assert_array_equal(run(lgd.CELL_VARCOEF_F64, u, k, 5, 0, 7), oracle.varcoef(u, k, 5))


@pytest.mark.parametrize("periodic", range(8))
@pytest.mark.parametrize("shape", [(5, 9, 33), (12, 7, 130)])
def test_fp64_any_boundary(periodic, shape):
    u, k = fields(shape, 2)
    edge = (0.3, 0.07, 0.0, 0.0)
    np.testing.assert_array_equal(run(lgd.CELL_VARCOEF_F64, u, k, 4, 0, periodic, edge),
                                  run(lgd.CELL_VARCOEF_F64, u, k, 4, 1, periodic, edge))


@pytest.mark.parametrize("scale", [0.0, 5e-324, 1e-308, 4.5e-308, 1e-300, 1e300, 8e307, np.inf])
def test_fp64_coefficients_at_the_ends_of_the_range(scale):
    u, k = fields((4, 6, 40), 3)
    k[1:3, 2:, ::3] = scale
    u[2, :, 5] = -u[2, :, 5]
    u[0] = 0.5
    np.testing.assert_array_equal(run(lgd.CELL_VARCOEF_F64, u, k, 2, 0, 7), run(lgd.CELL_VARCOEF_F64, u, k, 2, 1, 7))


@pytest.mark.parametrize("reach", [1, 9, 10, 30])
@pytest.mark.parametrize("bits", [3, 52])
def test_fp64_coefficients_far_apart(reach, bits):
    """The integer sum's condition met by all, some and none of a warp's
    faces; few significant bits (ties) and full significands."""
    rng = np.random.default_rng(reach)
    u = rng.random((6, 9, 40))
    k = np.ldexp(1.0 + np.floor(rng.random(u.shape) * 2.0 ** bits) * 2.0 ** -bits, rng.integers(-reach - 2, -1, u.shape))
    np.testing.assert_array_equal(run(lgd.CELL_VARCOEF_F64, u, k, 2, 0, 7), run(lgd.CELL_VARCOEF_F64, u, k, 2, 1, 7))


@pytest.mark.parametrize("periodic", [0, 5, 7])
@pytest.mark.parametrize("shape", SHAPES)
def test_fp32_ragged_rows(periodic, shape):
    """Three steps of sums of 14 terms below one: within 40 roundings."""
    u, k = (a.astype(np.float32) for a in fields(shape, 4))
    edge = (0.25, 0.05, 0.0, 0.0)
    np.testing.assert_allclose(run(lgd.CELL_VARCOEF_F32, u, k, 3, 0, periodic, edge),
                               run(lgd.CELL_VARCOEF_F32, u, k, 3, 1, periodic, edge), rtol=0, atol=40 * 2.0 ** -24)


@pytest.mark.parametrize("kind", ["zeros", "blocks", "both signs", "far apart", "one cell"])
@pytest.mark.parametrize("periodic", [0, 7])
def test_fp64_warps_that_fall_back(kind, periodic):
    """Grids whose threads march several planes (chunks of 8 here), where a warp
    computes planes as written after some that it did not: every bit that of
    variant 1, signs of zeros too."""
    shape = (100, 128, 128)
    rng = np.random.default_rng(6)
    u, k = fields(shape, 6)
    u[rng.random(shape) < 0.2] = 0.0
    u[rng.random(shape) < 0.2] *= -1.0              # and -0
    u[20:40, 20:60] = -0.0
    if kind == "zeros":
        k[rng.random(shape) < 0.5] = 0.0
    elif kind == "blocks":
        k[30:50, 10:70] = 0.0
        k[60:, :, 40:] = 0.0
    elif kind == "both signs":
        k[rng.random(shape) < 0.01] *= -1.0
    elif kind == "far apart":
        k[:, 40:] *= 2.0 ** -14
        k[13:, :, 70:] *= 2.0 ** -20
    else:
        k[51, 64, 77] = -0.05
    edge = (0.0, 0.07, 0.0, 0.0)
    a, b = (run(lgd.CELL_VARCOEF_F64, u, k, 3, variant, periodic, edge) for variant in (0, 1))
    np.testing.assert_array_equal(a.view(np.uint64), b.view(np.uint64))


@pytest.mark.parametrize("scale", [5e-324, 1e-308, 4.5e-308, 1e-300, 1.0, 1e300, 8e307, np.inf])
@pytest.mark.parametrize("bits", [2, 52])
def test_fp64_differences_of_u_at_the_ends_of_the_range(scale, bits):
    """The product's other operand: subnormal, overflowing and infinite
    differences, zeros of both signs, few significant bits (ties)."""
    rng = np.random.default_rng(bits)
    shape = (6, 9, 40)
    m = (1.0 + np.floor(rng.random(shape) * 2.0 ** bits) * 2.0 ** -bits) * rng.choice([-1.0, 1.0], shape)
    with np.errstate(over="ignore"):
        u = np.where(rng.random(shape) < 0.4, m * scale, m)
        u[2] = m[2] * scale
    u[rng.random(shape) < 0.1] = 0.0
    u[rng.random(shape) < 0.1] = -0.0
    k = np.ldexp(1.0 + np.floor(rng.random(shape) * 2.0 ** bits) * 2.0 ** -bits, rng.integers(-6, -2, shape))
    a, b = (run(lgd.CELL_VARCOEF_F64, u, k, 2, variant, 7) for variant in (0, 1))
    same = np.isnan(a) & np.isnan(b)                            # any NaN is a NaN
    np.testing.assert_array_equal(np.where(same, 0.0, a).view(np.uint64), np.where(same, 0.0, b).view(np.uint64))
