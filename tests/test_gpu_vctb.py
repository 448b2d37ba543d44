"""The two-step var-coef pass (csrc/k_vctb.cu, the default of FP32 tori whose
rows are a multiple of 16 bytes) against single steps, bit for bit: boxes cut
by the wrap in every axis, axes shorter than the halo, z chunks, an odd step
count."""
import numpy as np
import pytest

from libgeodecomp_gb300 import lgd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 4), (2, 3, 4), (3, 2, 56), (5, 60, 60), (9, 61, 64), (40, 59, 112),
                                   (33, 128, 116), (70, 16, 256), (11, 130, 8)])
@pytest.mark.parametrize("steps", [2, 7])
def test_two_steps_per_pass_equal_single_steps(shape, steps):
    rng = np.random.default_rng(sum(shape))
    u0 = rng.random(shape).astype(np.float32)
    k = (0.02 + 0.13 * rng.random(shape)).astype(np.float32)
    out, launches = [], []
    for depth in (0, 1):
        with lgd.Grid(lgd.CELL_VARCOEF_F32, shape, periodic=7) as g:
            g.set_time_block(depth)
            g.upload(0, u0)
            g.upload(1, k)
            n = g.launch_count()
            g.step(steps)
            launches.append(g.launch_count() - n)
            out.append(g.download(0))
    assert launches == [steps // 2 + steps % 2, steps]
    np.testing.assert_array_equal(out[0], out[1])
