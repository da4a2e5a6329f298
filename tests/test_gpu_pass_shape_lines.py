"""The lines at which a pass is cut up differently (pass_shape): chunks of 32 meshlets below 512 visible units, 64 from there,
128 from 1,024, 256 from 2,048, 512 from 4,096; 32 instances a warp below twice as many units as k_instances has blocks.
On both sides of each line, reached by batches of views of one scene whose cells are all visible, every view's draw set,
index regions and counters equal the oracle's float mirror."""
from types import SimpleNamespace

import numpy as np
import pytest

from parity_util import Harness, check_index_tiling, grid_matrices
from vgcut import engine, scenes
from vgcut.camera import Camera

pytestmark = pytest.mark.gpu

# (cells, views): their product is the number of visible units
LINES = [(73, 7), (64, 8), (27, 19),  # 511, 512, 513
         (93, 11), (64, 16),  # 1023, 1024
         (89, 23), (64, 32),  # 2047, 2048
         (91, 26), (74, 32), (103, 23),  # 2366, 2368, 2369: twice 148 multiprocessors of 8 blocks
         (117, 35), (128, 32), (100, 41)]  # 4095, 4096, 4100


@pytest.mark.parametrize("cells,views", LINES)
def test_both_sides(cells, views):
    n = cells * 128 - 5  # the last cell not full
    spec = SimpleNamespace(meshes=[scenes.icosphere_mesh(40, seed=2)], instances=[grid_matrices(n, 0.4, n)])
    h = Harness(spec, [dict(shadow=True)], max_meshlets=1 << 18, max_triangles=20_000_000, max_shadow=20_000_000,
                output_slots=views)
    side = np.ceil(np.sqrt(n)) * 0.4
    cam = Camera.perspective_look_at((side / 2, 2.0, -3.0), (side / 2, 0.0, side / 2), 60, 1920, 1080, 0.1, 5000.0)
    params = [engine.ViewParams(error_threshold=t, lod_blend=2.0, frustum_culling=False, shadow_sweep=(3.0, -9.0, 2.0),
                                fresh_state=True) for t in (1.5, 3.0)]
    want = [h.oracle(cam, p, state=[10000, 10000, 0, 0, 0, 0, 0, 0])[0] for p in params]
    batch = [engine.make_view(cam, engine.ViewParams(**{**params[k % 2].__dict__, "state_slot": k})) for k in range(views)]
    for graph in (False, True):
        h.vg.cut(batch, graph=graph)
        units, queued = 0, 0
        for k in range(views):
            s, o = h.vg.read_stats(k), want[k % 2]
            units, queued = units + s["visible_cells"], queued + s["meshlets_queued"]
            assert s["faults"] == 0 and s["rounds"] == o["rounds"] == 1
            for cut in (0, 1):
                got = [s["selected"][cut], s["drawn"][cut], s["survived"][cut], s["work"][cut], s["requested_indices"][cut]]
                assert got == o["counters"][2 + cut * 5:7 + cut * 5]
                entries = h.vg.draw_list(k, cut)
                keys = entries[:, [0, 1, 3]]
                expect = np.asarray(o["entries"][cut])
                assert np.array_equal(keys[np.lexsort(keys.T)], expect[np.lexsort(expect.T)]), (k, cut)
                check_index_tiling(entries, h.inst_slot, o["mesh_counts"], cut)
        assert units == cells * views
        assert queued > 512 * 2 * units  # more than a chunk of the largest size for each 64 instances
    h.vg.dispose()
