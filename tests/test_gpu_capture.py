"""Time steps that the caller captures into a CUDA graph on the handle's stream,
the grid's first steps among them: buffers made on first use must not end the
capture.  A replay gives what the same call gives outside a graph."""
import numpy as np
import pytest

from libgeodecomp_gb300 import lgd, workloads

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def fields(cell, shape):
    if cell == lgd.CELL_GOL_U8:
        return [workloads.gol_initial(shape[1], shape[0], seed=9)]
    rng = np.random.default_rng(9)
    return [rng.random(shape)] + ([0.02 + 0.1 * rng.random(shape)] if cell in (lgd.CELL_VARCOEF_F32, lgd.CELL_VARCOEF_F64) else [])


@pytest.mark.parametrize("cell,shape,periodic", [
    (lgd.CELL_GOL_U8, (80, 96), 3), (lgd.CELL_GOL_U8, (80, 101), 3), (lgd.CELL_GOL_U8, (33, 70), 0),
    (lgd.CELL_JACOBI7_F64, (9, 20, 33), 0), (lgd.CELL_JACOBI7_F32, (9, 20, 33), 0),
    (lgd.CELL_VARCOEF_F32, (9, 20, 32), 7), (lgd.CELL_VARCOEF_F64, (9, 20, 33), 7)])
def test_first_steps_captured(cell, shape, periodic):
    init = fields(cell, shape)
    out = []
    for captured in (True, False):
        with lgd.Grid(cell, shape, periodic=periodic) as g:
            for m, a in enumerate(init):
                g.upload(m, a)
            if captured:
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph, stream=torch.cuda.ExternalStream(g.stream())):
                    g.step(12)
                graph.replay()
                torch.cuda.synchronize()
            else:
                g.step(12)
            out.append(g.download(0))
            if captured:
                del graph
    np.testing.assert_array_equal(out[0], out[1])


def test_mma_sync_forward_captured():
    """The mma.sync path's buffers and packed weights, made in a capture."""
    from libgeodecomp_gb300 import surrogate
    shape = (3, 8, 32)
    u, k = (torch.rand((1,) + shape, device="cuda") for _ in range(2))
    out = []
    for captured in (True, False):
        with surrogate.SurrogateNet(shape) as net:
            net.set_params(surrogate.init_params(24, 1))
            net.set_variant(1)
            du = torch.zeros_like(u)
            torch.cuda.synchronize()
            if captured:
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph, stream=torch.cuda.ExternalStream(net.stream())):
                    net.forward(u, k, du)
                graph.replay()
                torch.cuda.synchronize()
                del graph
            else:
                net.forward(u, k, du)
                net.synchronize()
            out.append(du.cpu().numpy())
    np.testing.assert_array_equal(out[0], out[1])


@pytest.mark.parametrize("variant", [0, 1])
def test_packed_weights_of_a_graph_count_when_it_runs(variant):
    """A captured first use of a path that is not replayed packs nothing, and a
    captured update reaches the path that did not record it."""
    from libgeodecomp_gb300 import surrogate
    shape = (3, 8, 32)
    u, k, t = (torch.rand((1,) + shape, device="cuda") for _ in range(3))
    du, ref = torch.zeros_like(u), torch.zeros_like(u)
    torch.cuda.synchronize()
    with surrogate.SurrogateNet(shape, training=True) as net, surrogate.SurrogateNet(shape) as plain:
        net.set_variant(1 - variant)
        net.set_params(surrogate.init_params(24, 1))
        stream = torch.cuda.ExternalStream(net.stream())
        net.set_variant(variant)
        unused = torch.cuda.CUDAGraph()
        with torch.cuda.graph(unused, stream=stream):
            net.forward(u, k, du)
        del unused

        def compare():
            net.set_variant(variant)
            net.forward(u, k, du)
            plain.set_variant(variant)
            plain.set_params(net.get_params())
            plain.forward(u, k, ref)
            plain.synchronize()
            np.testing.assert_array_equal(du.cpu().numpy(), ref.cpu().numpy())

        compare()
        before = net.get_params()
        net.backward(t)
        net.set_variant(1 - variant)
        net.forward(u, k, du)
        update = torch.cuda.CUDAGraph()
        with torch.cuda.graph(update, stream=stream):
            net.adam(0.01)
        compare()                                   # captured only: nothing has changed
        update.replay()
        torch.cuda.synchronize()
        assert np.abs(net.get_params() - before).max() > 1e-3
        compare()
        del update
