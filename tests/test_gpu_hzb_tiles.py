"""The HZB tile kernel (64 x 64 tiles, 16 rows a warp, columns l and l + 32 a lane) and the one-block tail (levels of up
to 4,096 texels kept in shared memory): every mip equals the oracle's max reduction, bit for bit, at the edges of a
tile, of a warp's rows and of the tail's shared memory."""
import ctypes as C

import numpy as np
import pytest

import oracle as O
from parity_util import d2h, grid_matrices
from vgcut import engine, scenes
from vgcut.camera import Camera

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def vg():
    v = engine.VirtualGeometry()
    v.create_mesh(scenes.icosphere_mesh(4, seed=2), grid_matrices(4, 2.0, 3))
    yield v
    v.dispose()


# (height, width). Tails from level 5 (a cut's build) over 4,096 texels: (1100, 4100); from level 7 (a build of its
# own): (2049, 32767) - 17 x 256 texels; a single row and column; both sides of 32 and 64 columns, 16 and 64 rows
@pytest.mark.parametrize("shape", [(1, 1), (1, 64), (16, 31), (17, 33), (64, 64), (63, 65), (65, 63), (128, 129),
                                   (129, 5000), (5000, 3), (1, 32768), (1100, 4100), (1437, 2555), (2049, 32767)])
def test_mips_equal_the_oracle(vg, shape):
    import torch
    img = np.random.default_rng(shape[0] * 40009 + shape[1]).random(shape, dtype=np.float32)
    img[img < 0.1] = 0.0
    mips = _oracle_mips(img)
    d = torch.from_numpy(img).cuda()
    engine.check(engine.lib().vgc_hzb_build(vg.handle, 0, d.data_ptr(), shape[1], shape[0], 1, None))
    assert np.array_equal(d2h(vg.hzb_info(0)["data"], len(mips), np.float32), mips)
    cam = Camera.perspective_look_at((-6.0, 5.0, -6.0), (2.0, 0.0, 2.0), 60, 1920, 1080, 0.1, 100.0)
    v = engine.make_view(cam, engine.ViewParams(hzb=0), depth=(d.data_ptr(), shape[1], shape[0]))
    for cut in (vg.cut, lambda views: vg.cut_noalloc(views[0])):
        torch.cuda.synchronize()
        torch.as_tensor(_Mips(vg, len(mips)), device="cuda").fill_(-1.0)  # what the cut does not write shows
        torch.cuda.synchronize()
        cut([v])
        torch.cuda.synchronize()
        assert np.array_equal(d2h(vg.hzb_info(0)["data"], len(mips), np.float32), mips)


def _oracle_mips(img):
    """O.hzb_build with room for the chain of a single row, twice the image."""
    h, w = img.shape
    out = np.zeros(2 * img.size + 64, np.float32)
    levels, tables = C.c_uint32(), [(C.c_uint32 * 16)() for _ in range(3)]
    n = O.lib().vgo_hzb_build(O._f(img), w, h, O._f(out), len(out), C.byref(levels), *tables)
    assert n >= 0
    return out[:n]


class _Mips:
    def __init__(self, vg, n):
        self.__cuda_array_interface__ = dict(shape=(n,), typestr="<f4", data=(vg.hzb_info(0)["data"], False), version=3)
