"""The tensor-core kernels of the surrogate (C = 24; csrc/conv_tc.cu and
wgrad_tc.cu) at the sizes where they can go wrong: one, two and four rows per
tile (nx a multiple of 128, 64, 32), bands of y cut by the grid, one plane, z
chunks, several samples - forward pass and gradients against the FP64
reference and against the mma.sync path (variant 1)."""
import numpy as np
import pytest

from oracle import surrogate_ref as sr

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SHAPES = [(1, 4, 32), (2, 4, 128), (5, 20, 64), (3, 12, 96), (9, 8, 128), (34, 16, 32)]


def run(shape, variant, u, k, target, p, training):
    from libgeodecomp_gb300.surrogate import SurrogateNet
    batch = u.shape[0]
    with SurrogateNet(shape, batch=batch, channels=24, training=training) as net:
        net.set_params(p.astype(np.float32))
        net.set_variant(variant)
        assert net.uses_tensor_core_path() == (variant == 0)
        t = [torch.tensor(a, dtype=torch.float32, device="cuda").contiguous() for a in (u, k, target)]
        du = torch.empty_like(t[0])
        torch.cuda.synchronize()
        net.forward(t[0], t[1], du)
        if not training:
            net.synchronize()
            return du.cpu().numpy().astype(np.float64), None, None
        t[0].zero_()                        # the backward pass needs nothing of the caller's forward inputs
        torch.cuda.synchronize()
        loss = net.backward(t[2])
        return du.cpu().numpy().astype(np.float64), loss, net.get_grads().astype(np.float64)


def inputs(shape, batch, seed):
    rng = np.random.default_rng(seed)
    u = rng.random((batch,) + shape)
    k = 0.02 + 0.13 * rng.random((batch,) + shape)
    target = 0.05 * rng.standard_normal((batch,) + shape)
    p = sr.init_params(24, seed=seed + 1)
    p[-1] = 0.02
    return u, k, target, p


def layers(g):
    o = 0
    for ci, co in sr.layer_shapes(24):
        for size in (27 * ci * co, co):
            yield g[o:o + size]
            o += size


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("training", [False, True])
def test_forward(shape, training):
    u, k, target, p = inputs(shape, 1, sum(shape))
    ref, _ = sr.forward(p, u[0], k[0], 24)
    scale = np.linalg.norm(ref)
    tc = run(shape, 0, u, k, target, p, training)[0][0]
    ms = run(shape, 1, u, k, target, p, training)[0][0]
    assert np.linalg.norm(tc - ref) / scale < 3e-2
    assert np.linalg.norm(tc - ms) / scale < 1e-2


@pytest.mark.parametrize("shape", SHAPES)
def test_gradients(shape):
    u, k, target, p = inputs(shape, 1, 3 + sum(shape))
    loss_ref, g_ref = sr.loss_and_grad(p, u[0], k[0], target[0], 24)
    _, loss, g = run(shape, 0, u, k, target, p, True)
    _, loss_ms, g_ms = run(shape, 1, u, k, target, p, True)
    assert abs(loss - loss_ref) / loss_ref < 2e-2
    assert abs(loss - loss_ms) / loss_ms < 1e-2
    for a, b, c in zip(layers(g), layers(g_ref), layers(g_ms)):
        nb = np.linalg.norm(b) + 1e-30
        assert a @ b / (np.linalg.norm(a) * nb + 1e-30) > 0.995
        assert np.linalg.norm(a - b) / nb < 0.08
        assert np.linalg.norm(a - c) / nb < 2e-2


@pytest.mark.parametrize("shape,batch", [((6, 8, 64), 5), ((4, 12, 32), 3)])
def test_batches_are_sums_of_their_samples(shape, batch):
    """The mean loss of a batch is the mean of its samples', so is the gradient."""
    u, k, target, p = inputs(shape, batch, 17)
    du, loss, g = run(shape, 0, u, k, target, p, True)
    parts = [run(shape, 0, u[j:j + 1], k[j:j + 1], target[j:j + 1], p, True) for j in range(batch)]
    np.testing.assert_array_equal(du, np.concatenate([q[0] for q in parts]))
    np.testing.assert_allclose(loss, np.mean([q[1] for q in parts]), rtol=1e-5)
    mean = np.mean([q[2] for q in parts], axis=0)
    for a, b in zip(layers(g), layers(mean)):
        # the loss gradient is rounded to BF16 at another scale: 2^-8 relative
        # per voxel, averaged over the sums
        assert np.linalg.norm(a - b) / np.linalg.norm(b) < 1e-2


@pytest.mark.parametrize("order", [(0, 1), (1, 0)])
def test_changed_weights_reach_either_path(order):
    """A path that did not run while the parameters changed packs them when
    it does: the same output as a network that had them from the start."""
    from libgeodecomp_gb300.surrogate import SurrogateNet
    shape = (4, 8, 64)
    u, k, target, p = inputs(shape, 1, 3)
    t = [torch.tensor(a, dtype=torch.float32, device="cuda").contiguous() for a in (u, k, target)]
    du = torch.empty_like(t[0])
    torch.cuda.synchronize()
    with SurrogateNet(shape, channels=24, training=True) as net:
        net.set_variant(order[0])
        net.set_params(p.astype(np.float32))
        net.forward(t[0], t[1], du)
        net.backward(t[2])
        net.adam(0.01)
        net.set_variant(order[1])
        net.forward(t[0], t[1], du)
        net.synchronize()
        out, changed = du.cpu().numpy(), net.get_params()
    assert np.max(np.abs(changed - p)) > 5e-3
    with SurrogateNet(shape, channels=24) as net:
        net.set_variant(order[1])
        net.set_params(changed)
        net.forward(t[0], t[1], du)
        net.synchronize()
        np.testing.assert_array_equal(out, du.cpu().numpy())


@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("calls", [1, 3])
def test_backward_after_advance_is_about_its_last_call(variant, calls):
    """advance leaves what a forward pass of its last call would: the same loss
    and gradients (up to the order of the FP32 atomic sums, 1e-6 relative)."""
    from libgeodecomp_gb300.surrogate import SurrogateNet
    shape = (5, 12, 64)
    u, k, target, p = inputs(shape, 2, 8)
    before, v, kt, tt = (torch.tensor(a, dtype=torch.float32, device="cuda").contiguous() for a in (u, u, k, target))
    du = torch.empty_like(v)
    torch.cuda.synchronize()
    out = []
    for step in ("advance", "forward"):
        with SurrogateNet(shape, batch=2, channels=24, training=True) as net:
            net.set_params(p.astype(np.float32))
            net.set_variant(variant)
            if step == "advance":
                net.advance(v, kt, calls)
            else:
                net.advance(before, kt, calls - 1)
                net.forward(before, kt, du)
            loss = net.backward(tt)
            out.append((loss, net.get_grads().astype(np.float64)))
    np.testing.assert_array_equal(v.cpu().numpy(), (before + du).cpu().numpy())
    np.testing.assert_allclose(out[0][0], out[1][0], rtol=1e-6)
    for a, b in zip(layers(out[0][1]), layers(out[1][1])):
        assert np.linalg.norm(a - b) / np.linalg.norm(b) < 1e-5
