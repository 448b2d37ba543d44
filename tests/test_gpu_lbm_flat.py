"""The one-thread-per-cell step of the D3Q19 ensemble (csrc/lbm.cu) where its
blocks of 128 cells end, against the oracle (FP64, bit for bit) and against the
persistent kernel (FP32, bit for bit), and the device conversion of instances
larger than one staging chunk."""
import time

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


@pytest.mark.parametrize("kernel", ["flat", "persistent", "looped", "two steps"])
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("precision", [4, 8])
def test_infinite_velocities(precision, axis, kernel):
    """A density that is finite and a velocity component that overflows: 0 * u
    makes every moving direction a NaN, the directions across the component
    too, as in the oracle."""
    L = 6
    plus, minus = ((2, 3), (1, 4), (5, 6))[axis]        # E W, N S, T B
    f = np.tile(0.05 + 0.01 * np.arange(19.0)[:, None, None, None], (1, L, L, L))
    big = 3e38 if precision == 4 else 1.5e308
    # what cell (2, 2, 2) pulls: the source cell is the cell minus the direction
    for i, sign in ((plus, 1), (minus, -1)):
        src = [2, 2, 2]
        src[axis] -= sign                               # x, y, z
        f[i, src[2], src[1], src[0]] = sign * big
    with np.errstate(all="ignore"):
        ref = oracle.lbm(L, 1, 1.2, 0.05, f)
    assert np.isnan(ref[1:, 2, 2, 2]).all() or precision == 4
    with lgd.LbmEnsemble([L], [1.2], lid=0.05, precision=precision) as e:
        e.upload(0, f)
        if kernel == "persistent":
            e.set_config(2, 64, 1)
        if kernel == "two steps":
            e.set_time_block(2, 0, 1)
        if kernel == "looped":
            e.step_looped(1)
        else:
            e.step(2 if kernel == "two steps" else 1)
        out = e.download(0)
    if kernel == "two steps":
        with np.errstate(all="ignore"):
            ref = oracle.lbm(L, 2, 1.2, 0.05, f)
        if precision == 4:
            # the neighbours that pulled a NaN from the blown-up cell
            assert np.isnan(out[1:, 2, 2, 1]).all() and np.isnan(out[1:, 3, 2, 2]).all()
        else:
            np.testing.assert_array_equal(out, ref)
    elif precision == 4:
        assert np.isnan(out[1:, 2, 2, 2]).all()
        out[:, 2, 2, 2] = ref[:, 2, 2, 2] = 0.0
        assert np.isfinite(out[:, 0]).all()
    else:
        np.testing.assert_array_equal(out, ref)


def rounded_fma(a, b, c):
    """fl(a b + c) of FP32 numbers: the product is exact in FP64, and the sum's
    second rounding only matters next to a tie."""
    return np.float32(np.float64(a) * np.float64(b) + np.float64(c))


def test_fp32_relaxation_rounds_the_weighted_term():
    """FP32 rounds keep f + w x once for the weighted term and once for the sum:
    of the two FMAs this is the one with the smaller error (see relax)."""
    L, omega = 12, np.float32(1.3)
    rng = np.random.default_rng(9)
    w = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)[:, None, None, None]
    f = np.float32(w * (1 + 0.2 * rng.uniform(-1, 1, (19, L, L, L))))
    e = np.array([(0, 0, 0), (0, 1, 0), (1, 0, 0), (-1, 0, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (-1, 1, 0), (-1, -1, 0),
                  (1, 1, 0), (1, -1, 0), (-1, 0, 1), (-1, 0, -1), (1, 0, 1), (1, 0, -1), (0, 1, 1), (0, 1, -1), (0, -1, 1),
                  (0, -1, -1)])
    inner = slice(1, L - 1)
    p = np.array([f[i][1 - z:L - 1 - z, 1 - y:L - 1 - y, 1 - x:L - 1 - x] for i, (x, y, z) in enumerate(e)])
    p64 = p.astype(np.float64)
    rho, u = p64.sum(axis=0), np.tensordot(e.T, p64, axes=1)
    d = rho / 3 - 0.5 * (u * u).sum(axis=0)
    with lgd.LbmEnsemble([L], [float(omega)], lid=0.05, precision=4) as ens:
        ens.upload(0, f.astype(np.float64))
        ens.step(1)
        out = np.float32(ens.download(0))[:, inner, inner, inner]
    keep = np.float32(1) - omega
    for i in range(1, 19):
        wi = omega * np.float32(1 / 6 if i < 7 else 1 / 12)
        eu = np.tensordot(e[i], u, axes=1)
        x = np.float32(d + eu + 1.5 * eu * eu)
        one, other = rounded_fma(keep, p[i], wi * x), rounded_fma(wi, x, keep * p[i])
        # x has roundings of its own on the device: the two forms are told apart
        # where they differ, by which one the outputs lie nearer to
        differ = one != other
        near = np.abs(out[i].astype(np.float64) - one)[differ].sum(), np.abs(out[i].astype(np.float64) - other)[differ].sum()
        assert near[0] < near[1], i


@pytest.mark.parametrize("L", [2, 5, 9, 10, 14, 15])
def test_conversion_on_host_or_device(L):
    """Instances around the sizes up to which FP32 populations convert on the
    host (19 * 9^3 values down, 14^3 up)."""
    rng = np.random.default_rng(L)
    f = rng.uniform(-1, 1, (19, L, L, L))
    with lgd.LbmEnsemble([L, 3, L], [1.3, 1.0, 0.7], precision=4) as e:
        e.upload(2, f)
        np.testing.assert_array_equal(e.download(2), f.astype(np.float32).astype(np.float64))
        np.testing.assert_array_equal(e.download(0), oracle.lbm_rest(L).astype(np.float32).astype(np.float64))


@pytest.mark.parametrize("L", [3, 8])
def test_copies_of_small_fp32_instances(L):
    """They take no longer than 1.2 times FP64 ones, which need no conversion,
    and 0.3 ns a value (with a kernel each 1.3 to 1.6 times FP64's time)."""
    for _ in range(5):                      # again before it counts as slower
        best = {}
        for precision in (4, 8):
            with lgd.LbmEnsemble([L], [1.3], precision=precision) as e:
                f = e.download(0)
                times = []
                for _ in range(30):
                    t = time.perf_counter()
                    for _ in range(20):
                        e.upload(0, f)
                        e.download(0)
                    times.append(time.perf_counter() - t)
                best[precision] = min(times)
        if best[4] < 1.2 * best[8] + 20 * 2 * 19 * L ** 3 * 0.3e-9:
            return
    raise AssertionError(best)


@pytest.mark.parametrize("kernel", ["flat", "read-only", "persistent", "looped"])
def test_fp32_rounding_of_a_step(kernel):
    """One step of populations of both signs, every rounding restated: squares of
    u, the density's third, 1.5 (e . u)^2, the lid's share and the old population
    inside an FMA each; the other products rounded."""
    L, omega, lid = 12, np.float32(1.3), np.float32(0.05)
    f = np.random.default_rng(9).uniform(-1, 1, (19, L, L, L)).astype(np.float32)
    e = [(0, 0, 0), (0, 1, 0), (1, 0, 0), (-1, 0, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (-1, 1, 0), (-1, -1, 0), (1, 1, 0),
         (1, -1, 0), (-1, 0, 1), (-1, 0, -1), (1, 0, 1), (1, 0, -1), (0, 1, 1), (0, 1, -1), (0, -1, 1), (0, -1, -1)]
    z, y, x = np.meshgrid(*[np.arange(L)] * 3, indexing="ij")
    p = np.empty_like(f)
    for i, (ex, ey, ez) in enumerate(e):
        sx, sy, sz = x - ex, y - ey, z - ez
        inside = (sx >= 0) & (sx < L) & (sy >= 0) & (sy < L) & (sz >= 0) & (sz < L)
        back = f[e.index((-ex, -ey, -ez))]
        if ey == -1 and ex != 0:
            lidded = rounded_fma(np.float32(6) * np.float32(1 / 36), np.float32(ex) * lid, back)
            back = np.where(y == L - 1, lidded, back)
        p[i] = np.where(inside, f[i, sz % L, sy % L, sx % L], back)

    def total(*idx):
        s = p[idx[0]]
        for i in idx[1:]:
            s = s + p[i]
        return s

    rho = total(*range(19))
    ux = total(2, 9, 10, 13, 14) - total(3, 7, 8, 11, 12)
    uy = total(1, 7, 9, 15, 16) - total(4, 8, 10, 17, 18)
    uz = total(5, 11, 13, 15, 17) - total(6, 12, 14, 16, 18)
    assert all(a.dtype == np.float32 for a in (rho, ux, uy, uz))
    usq = rounded_fma(uz, uz, rounded_fma(ux, ux, uy * uy))
    d = rounded_fma(rho, np.float32(1 / 3), np.float32(-0.5) * usq)
    keep = np.float32(1) - omega
    ref = np.empty_like(f)
    ref[0] = rounded_fma(keep, p[0], omega * d)
    for i, (ex, ey, ez) in enumerate(e[1:], 1):
        eu = np.float32(ex) * ux + np.float32(ey) * uy + np.float32(ez) * uz
        w = omega * np.float32(1 / 6 if i < 7 else 1 / 12)
        ref[i] = rounded_fma(keep, p[i], w * rounded_fma(np.float32(1.5), eu * eu, d + eu))
    with lgd.LbmEnsemble([L], [float(omega)], lid=float(lid), precision=4) as ens:
        if kernel == "read-only":
            ens.set_variant(1)
        if kernel == "persistent":
            ens.set_config(4, 256, 4)
        ens.upload(0, f.astype(np.float64))
        ens.step_looped(1) if kernel == "looped" else ens.step(1)
        out = ens.download(0).astype(np.float32)
    np.testing.assert_array_equal(out, ref)


def test_table_of_a_large_ensemble_is_made_on_the_device():
    """Its 131072 entries (64 cavities of 64^3) took the host and the copy 1.3 ms of
    create's 1.8."""
    times = []
    for _ in range(40):
        t = time.perf_counter()
        e = lgd.LbmEnsemble([64] * 64, [1.2] * 64)
        times.append(time.perf_counter() - t)
        assert e.config() == (1, 128, 32)
        e.close()
    assert min(times) < 1.2e-3, times
