"""Packed Game of Life (csrc/k_golpack.cu, the default of calls of several
generations) against the oracle: widths around a word, a tile of 30 words and
a window that wraps onto itself, heights from one row over one tile to
several bands, torus and cube with dead and living edges, mixed axes, and a
step count that ends in a short pass."""
import numpy as np
import pytest

import oracle
from libgeodecomp_gb300 import lgd, workloads

pytestmark = pytest.mark.gpu


def run(c0, steps, periodic, edge=0.0, pack=True):
    with lgd.Grid(lgd.CELL_GOL_U8, c0.shape, periodic=periodic, edge=(edge, 0, 0, 0)) as g:
        if not pack:
            g.set_time_block(1)
        g.upload(0, c0)
        g.step(steps)
        return g.download(0)


SHAPES = [(1, 32), (5, 33), (40, 63), (2, 64), (129, 95), (33, 959), (70, 960), (64, 961), (513, 1001), (37, 1984),
          (1100, 2047), (3000, 40)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("steps", [37, 70])
def test_torus(shape, steps):
    c0 = workloads.gol_initial(shape[1], shape[0], seed=61)
    np.testing.assert_array_equal(run(c0, steps, 3), oracle.gol(c0, steps))


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("periodic,edge", [(0, 0.0), (0, 1.0), (1, 1.0), (2, 0.0)])
def test_cube_and_mixed_axes(shape, periodic, edge):
    """Against the byte-wise kernel, one launch per generation."""
    c0 = workloads.gol_initial(shape[1], shape[0], seed=62)
    np.testing.assert_array_equal(run(c0, 39, periodic, edge), run(c0, 39, periodic, edge, pack=False))


def test_bytes_other_than_0_and_1_keep_their_meaning():
    """Boards the byte-wise kernel served: a byte counts with its value."""
    c0 = workloads.gol_initial(101, 77, seed=63) * np.random.default_rng(1).integers(1, 4, (77, 101)).astype(np.uint8)
    for periodic in (0, 3):
        np.testing.assert_array_equal(run(c0, 20, periodic), run(c0, 20, periodic, pack=False))


@pytest.mark.parametrize("nx", [961, 1921, 1936, 1951, 1952, 2881, 2911, 3850])
@pytest.mark.parametrize("steps", [8, 33])
def test_last_partial_word_in_a_tiles_last_lane(nx, steps):
    """Rows that wrap and whose last, partial word is the one window of its tile
    that takes more than one word: 1921 .. 1951 cells, and every 960 more."""
    c0 = workloads.gol_initial(nx, 41, seed=64)
    np.testing.assert_array_equal(run(c0, steps, 3), oracle.gol(c0, steps))
    np.testing.assert_array_equal(run(c0, steps, 1), run(c0, steps, 1, pack=False))
