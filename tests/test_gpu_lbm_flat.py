"""The one-thread-per-cell step of the D3Q19 ensemble (csrc/lbm.cu) where its
blocks of 128 cells end, against the oracle (FP64, bit for bit) and against the
persistent kernel (FP32, bit for bit), and the device conversion of instances
larger than one staging chunk."""
import numpy as np
import pytest

import oracle
from libgeodecomp_gb300 import lgd

pytestmark = pytest.mark.gpu

# L^3 below, at and above multiples of 128; rows shorter and longer than a warp
EDGES = [2, 3, 4, 5, 8, 11, 16, 31, 32, 33]


@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("steps", [1, 6])
def test_flat_step_matches_oracle(variant, steps):
    omegas = [0.6 + 0.1 * j for j in range(len(EDGES))]
    with lgd.LbmEnsemble(EDGES, omegas, lid=0.05, precision=8) as e:
        e.set_variant(variant)
        e.step(steps)
        for j, L in enumerate(EDGES):
            np.testing.assert_array_equal(e.download(j), oracle.lbm(L, steps, omegas[j], 0.05), err_msg=str(L))


@pytest.mark.parametrize("edges", [EDGES, [64, 2, 65], [40, 80]])
def test_flat_step_equals_persistent_kernel(edges):
    omegas = [1.0 + 0.05 * j for j in range(len(edges))]
    with lgd.LbmEnsemble(edges, omegas, precision=4) as a, lgd.LbmEnsemble(edges, omegas, precision=4) as b:
        b.set_config(3, 128, 2)
        for n in (1, 4):
            a.step(n)
            b.step(n)
        for j in range(len(edges)):
            np.testing.assert_array_equal(a.download(j), b.download(j))


def test_conversion_beyond_one_chunk():
    """19 * 80^3 values pass the staging buffer in two chunks each way."""
    rng = np.random.default_rng(2)
    f = rng.random((19, 80, 80, 80)).astype(np.float32).astype(np.float64)
    with lgd.LbmEnsemble([80], [1.3], precision=4) as e:
        e.upload(0, f)
        np.testing.assert_array_equal(e.download(0), f)


@pytest.mark.parametrize("omega", [1.0, 0.5, 1.999])
@pytest.mark.parametrize("scale", [1.0, 2.0 ** -520, 1e-300, 1e160, 0.0])
def test_fp64_products_at_the_ends_of_the_range(scale, omega):
    """Populations whose products are zero, subnormal or overflow (the cell is
    then computed with FP64 multiplications), mixed with ordinary ones; the
    persistent kernel multiplies in FP64 throughout."""
    rng = np.random.default_rng(7)
    f = rng.random((19, 7, 7, 7)) * np.where(rng.random((1, 7, 7, 7)) < 0.5, scale, 1.0) * rng.choice([-1.0, 1.0], (19, 7, 7, 7))
    f[:, :2] = 0.0
    out = []
    for persistent in (False, True):
        with lgd.LbmEnsemble([7], [omega], lid=0.05, precision=8) as e:
            if persistent:
                e.set_config(2, 64, 1)
            e.upload(0, f)
            e.step(3)
            out.append(e.download(0))
    np.testing.assert_array_equal(out[0], out[1])
