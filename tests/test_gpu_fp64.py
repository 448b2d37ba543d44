"""The IEEE FP64 Jacobi kernel (csrc/k_fp64.cu) against the oracle, bit for
bit, at the sizes and values where it can go wrong: planes around one CTA of
128 cells, z chunks that end short, values that leave the integer product's
range, and non-zero edges."""
import numpy as np
import pytest

import oracle
from libgeodecomp_gb300 import lgd, workloads

pytestmark = pytest.mark.gpu


def run(u0, steps, edge=0.0, periodic=0):
    with lgd.Grid(lgd.CELL_JACOBI7_F64, u0.shape, periodic=periodic, edge=(edge, 0, 0, 0)) as g:
        g.upload(0, u0)
        g.step(steps)
        return g.download(0)


@pytest.mark.parametrize("shape", [(1, 1, 127), (2, 16, 8), (3, 43, 3), (17, 1, 129), (9, 33, 31), (130, 96, 64)])
@pytest.mark.parametrize("edge", [0.0, -0.5])
def test_shapes(shape, edge):
    u0 = workloads.jacobi_initial(shape[2], shape[1], shape[0], seed=51)
    np.testing.assert_array_equal(run(u0, 5, edge), oracle.jacobi7(u0, 5, edge=edge))


@pytest.mark.parametrize("scale", [1e-323, 3e-308, 1e-300, 1.0, 1e300, 2e307])
def test_value_ranges(scale):
    """Subnormals, the ends of the exponent range, negative values, zeros and
    sums whose significand makes the product a tie."""
    rng = np.random.default_rng(5)
    u0 = (rng.uniform(-1.0, 1.0, (7, 12, 40)) * scale).astype(np.float64)
    u0[2] = 0.0
    u0[4] = scale * 0.25
    with np.errstate(over="ignore", invalid="ignore"):
        ref = oracle.jacobi7(u0, 3)
    out = run(u0, 3)
    np.testing.assert_array_equal(out.view(np.uint64), ref.view(np.uint64))


@pytest.mark.parametrize("reach", [0, 5, 6, 7, 40])
@pytest.mark.parametrize("shape", [(3, 9, 33), (5, 6, 128)])
def test_exponent_distances(reach, shape):
    """The integer sum's condition met by all, some and none of a warp's
    cells, with few significant bits (ties) and full significands, of one
    sign and of both."""
    rng = np.random.default_rng(reach)
    for bits, both in [(3, False), (52, False), (52, True)]:
        m = 1.0 + np.floor(rng.random(shape) * 2.0 ** bits) * 2.0 ** -bits
        u0 = np.ldexp(m, rng.integers(0, reach + 1, shape))
        if both:
            u0 *= np.where(rng.random(shape) < 0.02, -1.0, 1.0)
        np.testing.assert_array_equal(run(u0, 1).view(np.uint64), oracle.jacobi7(u0, 1).view(np.uint64))
        np.testing.assert_array_equal(run(-u0, 4), oracle.jacobi7(-u0, 4))


@pytest.mark.parametrize("shape", [(1, 1, 127), (3, 2, 1), (2, 16, 8), (17, 1, 129), (9, 33, 31), (130, 96, 64)])
def test_torus(shape):
    u0 = workloads.jacobi_initial(shape[2], shape[1], shape[0], seed=52)
    np.testing.assert_array_equal(run(u0, 5, periodic=7), oracle.jacobi7(u0, 5, torus=True))


@pytest.mark.parametrize("periodic", [1, 2, 3, 4, 5, 6])
@pytest.mark.parametrize("shape", [(4, 7, 33), (2, 3, 40)])
def test_some_axes_wrap(periodic, shape):
    """A grid that wraps along some axes only, against one extended along
    them by as many cells as steps."""
    steps = 3
    u0 = workloads.jacobi_initial(shape[2], shape[1], shape[0], seed=53)
    pad = [(steps, steps) if periodic >> axis & 1 else (0, 0) for axis in (2, 1, 0)]
    inner = tuple(slice(a, a + n) for (a, _), n in zip(pad, shape))
    ref = oracle.jacobi7(np.pad(u0, pad, mode="wrap"), steps, edge=0.25)[inner]
    np.testing.assert_array_equal(run(u0, steps, edge=0.25, periodic=periodic), ref)


@pytest.mark.parametrize("periodic", [0, 7])
@pytest.mark.parametrize("edge", [0.0, -0.0, 0.25])
def test_empty_parts(periodic, edge):
    """Zeros of either sign next to each other, to subnormals and to a hot spot:
    the sign of every zero sum, too (grids whose threads march eight planes)."""
    shape = (100, 128, 128)
    rng = np.random.default_rng(8)
    u0 = np.zeros(shape)
    u0[50, 64, 64] = 1.0
    u0[20:30, 10:20] = -0.0
    u0[40:44, :, 30:33] = np.where(rng.random((4, 128, 3)) < 0.5, -0.0, 0.0)
    u0[70:, 100:, 100:] = rng.integers(-2, 3, (30, 28, 28)) * 5e-324
    out = []
    for variant in (0, 2):
        with lgd.Grid(lgd.CELL_JACOBI7_F64, shape, periodic=periodic, edge=(edge, 0, 0, 0)) as g:
            g.set_variant(variant)
            g.upload(0, u0)
            g.step(4)
            out.append(g.download(0).view(np.uint64))
    np.testing.assert_array_equal(out[0], out[1])
