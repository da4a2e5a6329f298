"""How a pass is cut up follows the visible units (k_instances: 32 or 64 instances a warp, chunks of 32..512 meshlets):
the draw sets and counters must equal the oracle's float mirror on both sides of every line, and when a launch of small
chunks asks for more than the meshlet queue holds (its items are tested in place)."""
from types import SimpleNamespace

import numpy as np
import pytest

from parity_util import Harness, grid_matrices
from vgcut import engine, scenes
from vgcut.camera import Camera

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mesh():
    return scenes.icosphere_mesh(24, seed=2)


# cells of 128 instances: one piece and one more of either size, a cell and one more; 16 / 17 cells (chunks of 32 / 64
# meshlets), 32 / 33 and 255 / 256 (64 / 128, 256 / 512)
@pytest.mark.parametrize("n", [1, 31, 32, 33, 64, 65, 127, 128, 129, 2048, 2049, 4096, 4097, 32640, 32768])
def test_instances_on_both_sides(mesh, n):
    spec = SimpleNamespace(meshes=[mesh], instances=[grid_matrices(n, 2.0, n)])
    h = Harness(spec, [dict(shadow=True)], max_meshlets=1 << 20, max_triangles=40_000_000, max_shadow=40_000_000)
    side = np.ceil(np.sqrt(n)) * 2.0
    cam = Camera.perspective_look_at((-6.0, 5.0, -6.0), (side / 2, 0.0, side / 2), 60, 1920, 1080, 0.1, 5000.0)
    for graph in (False, True):
        lists, res = h.compare(cam, engine.ViewParams(error_threshold=1.6, frustum_culling=False,
                                                      shadow_sweep=(3.0, -9.0, 2.0), fresh_state=True), graph=graph)
        assert len(lists[0]) > 0 and len(lists[1]) > 0
    h.vg.dispose()


def test_queue_overflow_with_small_chunks(mesh):
    n = 100_000
    spec = SimpleNamespace(meshes=[mesh], instances=[grid_matrices(n, 1.5, 11)])
    h = Harness(spec, [{}], max_meshlets=1 << 23, max_triangles=300_000_000)
    side = np.ceil(np.sqrt(n)) * 1.5
    cam = Camera.perspective_look_at((side / 2, 60.0, side / 2 + 1.0), (side / 2, 0.0, side / 2), 60, 1920, 1080, 0.1,
                                     5000.0)
    p = engine.ViewParams(error_threshold=0.02, frustum_culling=False, fresh_state=True)
    for _ in range(2):  # the first call overflows the fresh queue, which grows before the second
        lists, res = h.compare(cam, p)
    # 782 cells: chunks of 64 meshlets, of which a fresh queue holds 65,536
    assert h.vg.last_stats["meshlets_queued"] > 65_536 * 64
    h.vg.dispose()
