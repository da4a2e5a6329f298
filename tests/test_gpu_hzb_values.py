"""Depth images with the values a maximum treats specially: NaN texels (fmaxf drops them; a footprint of NaN alone stays
NaN), infinities, zeros of both signs and denormals. Every mip equals the maximum that numpy's fmax gives, by value, and
mip 0 the image bit for bit, through the tile kernel and through the strip stream of a cut."""
import numpy as np
import pytest

from parity_util import d2h, grid_matrices
from vgcut import engine, scenes
from vgcut.camera import Camera

pytestmark = pytest.mark.gpu


def _mips(img):
    out, lw = [img], img
    while lw.shape != (1, 1):
        h, w = lw.shape
        rows = np.fmax(lw[0::2], lw[np.minimum(np.arange(0, h, 2) + 1, h - 1)])
        lw = np.fmax(rows[:, 0::2], rows[:, np.minimum(np.arange(0, w, 2) + 1, w - 1)])
        out.append(lw)
    return out


@pytest.mark.parametrize("shape", [(1, 1), (33, 65), (64, 128), (130, 257), (540, 960)])
def test_special_values(shape):
    import torch
    rng = np.random.default_rng(shape[1])
    img = rng.random(shape, dtype=np.float32)
    kinds = rng.integers(0, 40, shape)
    for k, v in enumerate((np.nan, np.inf, -np.inf, 0.0, -0.0, 1e-42)):
        img[kinds == k] = v
    img[:16, :16] = np.nan  # whole footprints
    want = _mips(img)
    vg = engine.VirtualGeometry(max_meshlets=1 << 10)
    vg.create_mesh(scenes.icosphere_mesh(4, seed=2), grid_matrices(4, 2.0, 3))
    cam = Camera.perspective_look_at((-6.0, 5.0, -6.0), (2.0, 0.0, 2.0), 60, 1920, 1080, 0.1, 100.0)
    d = torch.from_numpy(img).cuda()
    view = engine.make_view(cam, engine.ViewParams(hzb=0), depth=(d.data_ptr(), shape[1], shape[0]))
    total = sum(m.size for m in want)
    for build in (lambda: engine.check(engine.lib().vgc_hzb_build(vg.handle, 0, d.data_ptr(), shape[1], shape[0], 1, None)),
                  lambda: vg.cut([view]), lambda: vg.cut_noalloc(view)):
        torch.cuda.synchronize()
        build()
        torch.cuda.synchronize()
        got = d2h(vg.hzb_info(0)["data"], total, np.float32)
        assert np.array_equal(got[:img.size].view(np.uint32), img.ravel().view(np.uint32))
        assert np.array_equal(got, np.concatenate([m.ravel() for m in want]), equal_nan=True)
    vg.dispose()
