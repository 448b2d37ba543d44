"""The default kernel is not the slower one where another can be selected for
the same call: the least of several timings each, with room for their spread, and
measured again before it counts as slower."""
import time

import numpy as np
import pytest

from libgeodecomp_gb300 import lgd, workloads

pytestmark = pytest.mark.gpu


def holds(measure, condition, tries=5):
    """Whether one of several measurements meets the condition."""
    seen = []
    for _ in range(tries):
        seen.append(measure())
        if condition(*seen[-1]):
            return True
    print(seen)
    return False


def least(grid, steps, setups, rounds=5):
    """Seconds per call of steps steps, the least of rounds timings, for each setup in turn."""
    best = [float("inf")] * len(setups)
    for _ in range(rounds):
        for i, setup in enumerate(setups):
            setup(grid)
            grid.step(steps)
            grid.synchronize()
            t = time.perf_counter()
            grid.step(steps)
            grid.synchronize()
            best[i] = min(best[i], time.perf_counter() - t)
    return best


@pytest.mark.parametrize("kind", ["zeros", "blocks", "both signs"])
def test_fp64_varcoef_of_any_coefficients(kind):
    """Against the pair kernel, whose time does not depend on them."""
    shape = (128, 128, 128)
    rng = np.random.default_rng(1)
    k = 0.02 + 0.13 * rng.random(shape)
    if kind == "zeros":
        k[rng.random(shape) < 0.5] = 0.0
    elif kind == "blocks":
        k[:, 64:] = 0.0
        k[64:, :, :32] = 0.0
    else:
        k -= 0.08
    with lgd.Grid(lgd.CELL_VARCOEF_F64, shape, periodic=7) as g:
        g.upload(0, rng.random(shape))
        g.upload(1, k)
        assert holds(lambda: least(g, 20, [lambda g: g.set_variant(0), lambda g: g.set_variant(2)]), lambda default, pair: default < 1.15 * pair)


@pytest.mark.parametrize("shape", [(1, 2048, 4096), (256, 2, 4096), (3000, 64, 64), (256, 256, 256), (40, 33, 64)])
def test_fp32_varcoef_of_any_shape(shape):
    """Two steps per pass where that is the faster, against single steps."""
    rng = np.random.default_rng(2)
    with lgd.Grid(lgd.CELL_VARCOEF_F32, shape, periodic=7) as g:
        g.upload(0, rng.random(shape))
        g.upload(1, 0.1 * rng.random(shape))
        assert holds(lambda: least(g, 40, [lambda g: g.set_time_block(0), lambda g: g.set_time_block(1)]), lambda default, single: default < 1.1 * single)


@pytest.mark.parametrize("shape,steps", [((1, 1000000), 6), ((4, 1000000), 8), ((8192, 16384), 6), ((8192, 16384), 12),
                                         ((1024, 1024), 6), ((16384, 16384), 8)])
def test_gol_calls_of_a_few_generations(shape, steps):
    """Packed rows where packing pays, against the bit-sliced passes over bytes."""
    board = (np.random.default_rng(3).integers(0, 3, shape, dtype=np.uint8) == 0).astype(np.uint8)
    with lgd.Grid(lgd.CELL_GOL_U8, shape, periodic=3) as g:
        g.upload(0, board)
        assert holds(lambda: least(g, steps, [lambda g: g.set_time_block(0), lambda g: g.set_time_block(16)], rounds=9), lambda default, passes: default < 1.12 * passes)


@pytest.mark.parametrize("exact", [False, True])
def test_fp64_sell_steps_grow_with_the_rows(exact):
    """A step's CTAs spread over the SMs: half as many rows again never take
    more than 30% longer among small matrices (piled up on some SMs they took 50%)."""
    rows = (20000, 30000, 40000, 60000, 90000)

    def measure():
        times = []
        for n in rows:
            g = lgd.SellGrid.from_csr(n, *workloads.powerlaw_graph(n, seed=1), 32, 256, exact=exact)
            g.upload(np.random.default_rng(0).random(n))
            times += least(g, 200, [lambda g: None])
            g.close()
        return times

    assert holds(measure, lambda a, b, c, d, e: b < 1.3 * a and d < 1.3 * c and e < 1.3 * d)


@pytest.mark.parametrize("kind", ["hot spot", "both signs", "uniform"])
@pytest.mark.parametrize("periodic", [0, 7])
def test_fp64_jacobi_of_any_field(kind, periodic):
    """Against the register kernel, whose time does not depend on the values."""
    n = 512 if kind == "hot spot" else 256
    shape = (n, n, n)
    rng = np.random.default_rng(5)
    u = np.zeros(shape) if kind == "hot spot" else rng.random(shape) - (0.5 if kind == "both signs" else 0.0)
    u[n // 2, n // 2, n // 2] = 1.0
    with lgd.Grid(lgd.CELL_JACOBI7_F64, shape, periodic=periodic) as g:
        g.upload(0, u)
        assert holds(lambda: least(g, 5, [lambda g: g.set_variant(0), lambda g: g.set_variant(5)]), lambda default, register: default < 1.03 * register)
