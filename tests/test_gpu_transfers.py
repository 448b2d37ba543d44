"""Host and device copies of rows that do not fill their pitch: the staged
dense copy and the row kernel (csrc/api.cu) return what was sent, for every
element size, odd row lengths, and grids of more than one staging chunk."""
import ctypes

import numpy as np
import pytest

from libgeodecomp_gb300 import lgd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cell,shape", [(lgd.CELL_GOL_U8, (5, 1)), (lgd.CELL_GOL_U8, (7, 1001)),
                                        (lgd.CELL_GOL_U8, (3, 1002)), (lgd.CELL_GOL_U8, (70001, 1003)),
                                        (lgd.CELL_JACOBI7_F32, (3, 5, 33)), (lgd.CELL_JACOBI7_F64, (2, 7, 17)),
                                        (lgd.CELL_JACOBI7_F64, (40, 64, 4097))])
def test_upload_download(cell, shape):
    rng = np.random.default_rng(3)
    a = rng.integers(0, 2, shape).astype(np.uint8) if cell == lgd.CELL_GOL_U8 else rng.random(shape)
    with lgd.Grid(cell, shape) as g:
        a = a.astype(g.members[0])
        g.upload(0, a)
        np.testing.assert_array_equal(g.download(0), a)


@pytest.mark.parametrize("cell,shape", [(lgd.CELL_GOL_U8, (9, 1001)), (lgd.CELL_VARCOEF_F32, (3, 5, 33)),
                                        (lgd.CELL_VARCOEF_F64, (2, 7, 17)), (lgd.CELL_JACOBI7_F32, (2, 3, 32))])
def test_device_copies(cell, shape):
    torch = pytest.importorskip("torch")
    with lgd.Grid(cell, shape) as g:
        a = torch.from_numpy(np.random.default_rng(4).integers(0, 2, shape).astype(g.members[0])).cuda()
        b = torch.empty_like(a)
        torch.cuda.synchronize()
        for name, t in (("lgd_gpu_upload_device", a), ("lgd_gpu_download_device", b)):
            fn = getattr(lgd.lib(), name)
            fn.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_void_p, ctypes.c_size_t]
            lgd.check(fn(g._h, 0, 0, t.data_ptr(), t.numel() * t.element_size()))
        np.testing.assert_array_equal(b.cpu().numpy(), a.cpu().numpy())
        np.testing.assert_array_equal(g.download(0), a.cpu().numpy())
