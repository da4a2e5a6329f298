"""Rounds 1 and 2 of a cut that overflows its index capacity (k_retry: four phases a round in one kernel; after a
launch that redid a cut, kernels of their own): draw sets,
counters, arguments and controller state equal the oracle's float mirror, for views that settle in different rounds of
one launch, and when the meshlet queue overflows in a retried round too."""
import ctypes as C
import time
from types import SimpleNamespace

import numpy as np
import pytest

from parity_util import Harness, grid_matrices, key_set
from vgcut import engine, scenes
from vgcut.camera import Camera

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mesh():
    return scenes.icosphere_mesh(24, seed=2)


def _camera(n, spacing, high=5.0):
    side = np.ceil(np.sqrt(n)) * spacing
    return Camera.perspective_look_at((-6.0, high, -6.0), (side / 2, 0.0, side / 2), 60, 1920, 1080, 0.1, 5000.0)


# cells of 128 instances; one unit and one more, several blocks' worth
@pytest.mark.parametrize("n", [1, 128, 129, 4097])
@pytest.mark.parametrize("share", [0.7, 0.05])  # of the index capacity the cut asks for: one round more, or two
def test_rounds_equal_the_oracle(mesh, n, share):
    spec = SimpleNamespace(meshes=[mesh], instances=[grid_matrices(n, 2.0, n)])
    p = engine.ViewParams(error_threshold=0.5, frustum_culling=False, fresh_state=True)
    cam = _camera(n, 2.0)
    whole = Harness(spec, [{}], max_meshlets=1 << 20, max_triangles=80_000_000)
    _, res = whole.compare(cam, p)
    wanted = whole.vg.last_stats["requested_indices"][0] // 3
    whole.vg.dispose()
    assert res["rounds"] == 1 and wanted > 100
    h = Harness(spec, [{}], max_meshlets=1 << 20, max_triangles=max(1, int(wanted * share)))
    for graph in (False, False, True, True):  # a launch after one that redid a cut has the rounds' own kernels
        _, res = h.compare(cam, p, graph=graph)
        assert res["rounds"] >= 2
    h.vg.dispose()


def test_views_of_one_launch_settle_in_their_own_round(mesh):
    n = 2049
    spec = SimpleNamespace(meshes=[mesh], instances=[grid_matrices(n, 2.0, n)])
    h = Harness(spec, [{}], max_meshlets=1 << 20, max_triangles=150_000)
    cam = _camera(n, 2.0)
    params = [engine.ViewParams(error_threshold=t, frustum_culling=False, fresh_state=True, state_slot=k)
              for k, t in enumerate((0.25, 64.0, 1.0, 4.0, 0.25, 16.0))]
    alone, rounds = [], []
    for p in params:
        lists, res = h.compare(cam, p)
        alone.append(key_set(lists[0], (0, 1, 3)))
        rounds.append(res["rounds"])
    assert len(set(rounds)) >= 2
    views = [engine.make_view(cam, p) for p in params]
    for graph in (False, False, True, True):
        h.vg.cut(views, graph=graph)
        for k in range(len(views)):
            s = h.vg.read_stats(k)
            assert s["rounds"] == rounds[k] and s["faults"] == 0
            assert key_set(h.vg.draw_list(k, 0), (0, 1, 3)) == alone[k]
    h.vg.dispose()


def test_queue_overflows_in_a_retried_round(mesh):
    """The cut without allocation has a queue of 49,152 spans; the last round of this one hands over more."""
    n = 100_000
    spec = SimpleNamespace(meshes=[mesh], instances=[grid_matrices(n, 1.5, 11)])
    h = Harness(spec, [{}], max_meshlets=1 << 23, max_triangles=120_000_000)
    side = np.ceil(np.sqrt(n)) * 1.5
    cam = Camera.perspective_look_at((side / 2, 60.0, side / 2 + 1.0), (side / 2, 0.0, side / 2), 60, 1920, 1080, 0.1,
                                     5000.0)
    p = engine.ViewParams(error_threshold=0.02, frustum_culling=False, fresh_state=True)
    lists, res = h.compare(cam, p)
    want = h.vg.read_stats(0)
    assert res["rounds"] >= 2 and want["work"][0] > 49_152
    for _ in range(2):
        h.vg.cut_noalloc(engine.make_view(cam, p), slot=1)
        got = h.vg.read_stats(1)
        for k in ("rounds", "selected", "drawn", "requested_indices", "work", "faults", "effective_threshold"):
            assert got[k] == want[k], k
        assert key_set(h.vg.draw_list(1, 0), (0, 1, 3)) == key_set(lists[0], (0, 1, 3))
    h.vg.dispose()


@pytest.mark.parametrize("limit_us", [2000, 20000])
def test_wait_gives_up(mesh, limit_us):
    """The wait for a phase that nothing completes ends at its limit with a fault; the context then cuts exactly."""
    spec = SimpleNamespace(meshes=[mesh], instances=[grid_matrices(33, 2.0, 1)])
    h = Harness(spec, [{}])
    faults = C.c_uint32()
    t = time.perf_counter()
    engine.check(engine.lib().vgc_debug_retry_probe(h.vg.handle, limit_us, C.byref(faults)))
    assert faults.value == 2 and limit_us * 1e-6 <= time.perf_counter() - t < 2.0
    h.compare(_camera(33, 2.0), engine.ViewParams(error_threshold=1.0, fresh_state=True))
    h.vg.dispose()
