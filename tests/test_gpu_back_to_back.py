"""Launch sequences one behind the other on one stream, without the host waiting between them: other cameras, other view
counts, other scenes' worth of visible units, plain launches, graphs and the cut without allocation in turn. Every draw
set equals that of the same cut with the device idle before and after."""
import ctypes as C

import numpy as np
import pytest

from parity_util import grid_matrices, key_set
from vgcut import engine, scenes
from vgcut.camera import Camera

pytestmark = pytest.mark.gpu


def test_sequences_one_behind_the_other():
    import torch
    vg = engine.VirtualGeometry(max_meshlets=1 << 15, output_slots=40)
    vg.create_mesh(scenes.icosphere_mesh(24, seed=2), grid_matrices(4000, 2.0, 5))
    vg.create_mesh(scenes.icosphere_mesh(8, seed=3), grid_matrices(700, 5.0, 6))
    rng = np.random.default_rng(4)

    def view(k):
        at = rng.uniform(0.0, 120.0, 2)
        cam = Camera.perspective_look_at((at[0], 3.0 + 9.0 * (k % 3), at[1]), tuple(rng.uniform(0.0, 120.0, 3) * (1, 0, 1)),
                                         35 + 20 * (k % 4), 1920, 1080, 0.1, 5000.0)
        return engine.make_view(cam, engine.ViewParams(error_threshold=float(rng.uniform(0.6, 6.0)), fresh_state=True,
                                                       frustum_culling=k % 5 != 0, state_slot=k))

    views = [view(k) for k in range(40)]
    want = []
    for k, v in enumerate(views):
        vg.cut([v], first_slot=k)
        torch.cuda.synchronize()
        want.append(key_set(vg.draw_list(k, 0), (0, 1, 3)))
    assert len(set(map(len, want))) > 20
    st = torch.cuda.Stream()
    sizes = (1, 7, 2, 16, 1, 4, 3, 5, 1)  # a batch of its own for each size: no call waits for the one before
    for order in range(4):
        with torch.cuda.stream(st):
            torch.cuda._sleep(4_000_000)  # the whole train is queued before it starts
        k = 0
        for i, n in enumerate(sizes):
            if n == 1 and (i + order) % 2:
                vg.cut_noalloc(views[k], slot=k, stream=st.cuda_stream)
            else:
                vg.cut(views[k:k + n], first_slot=k, stream=st.cuda_stream, graph=n > 1)
            k += n
        torch.cuda.synchronize()
        for j in range(k):
            assert vg.read_stats(j)["faults"] == 0 and key_set(vg.draw_list(j, 0), (0, 1, 3)) == want[j], (order, j)
    vg.dispose()


@pytest.mark.parametrize("shape", [(37, 41), (270, 481), (1080, 1920)])
def test_hzb_behind_the_kernel_that_draws_its_image(shape):
    """An image drawn by a kernel just before its HZB is built: the new texels, not those of the image before."""
    import torch
    vg = engine.VirtualGeometry()
    vg.create_mesh(scenes.icosphere_mesh(4, seed=2), grid_matrices(4, 2.0, 3))
    img = torch.zeros(shape, device="cuda")
    for k in range(20):
        img.fill_(0.25 + k / 64.0)
        engine.check(engine.lib().vgc_hzb_build(vg.handle, 0, img.data_ptr(), shape[1], shape[0], 1,
                                                C.c_void_p(torch.cuda.current_stream().cuda_stream or 1)))
        img.fill_(0.0)
        torch.cuda.synchronize()
        info = vg.hzb_info(0)
        total = info["offset"][info["levels"] - 1] + 1
        mips = torch.as_tensor(_Mips(info["data"], total), device="cuda")
        assert bool((mips == 0.25 + k / 64.0).all())
    vg.dispose()


class _Mips:
    def __init__(self, data, n):
        self.__cuda_array_interface__ = dict(shape=(n,), typestr="<f4", data=(data, False), version=3)
