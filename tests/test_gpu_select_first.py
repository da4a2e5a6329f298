"""A context's first selectCut takes no more memory than the call needs and page-locks none; its later calls, with a kept
workspace that grows with them and, after many, page-locked pieces, return the same bytes."""
import numpy as np
import pytest

from vgcut import engine, scenes

pytestmark = pytest.mark.gpu

ONE = np.eye(4, dtype=np.float32).reshape(1, 16)


def _call(vg, mesh, n):
    vm = np.tile(np.eye(4).reshape(1, 16), (n, 1))
    vm[:, 14] = -np.linspace(2.0, 40.0, n)
    return vg.select_cut(mesh.slot, vm, 900.0, 0.1, np.ones(n), 1.0, 2.0)


def _bytes(mesh, n):
    return (n * 19 * 4 + 255 & ~255) + 2 * n * mesh.data.meshlet_count


@pytest.mark.parametrize("subdivision,n", [(8, 1), (24, 9), (160, 40)])
def test_first_call_takes_what_it_needs(subdivision, n):
    vg = engine.VirtualGeometry(max_meshlets=1 << 10)
    mesh = vg.create_mesh(scenes.icosphere_mesh(subdivision), ONE)
    vg.debug_cells_device()  # the scene's upload
    before = vg.footprint()
    lo, hi = _call(vg, mesh, n)
    assert vg.footprint() - before == _bytes(mesh, n)
    for _ in range(20):  # the pieces come with the 17th call
        again = _call(vg, mesh, n)
        assert np.array_equal(again[0], lo) and np.array_equal(again[1], hi)
    assert vg.footprint() - before == _bytes(mesh, n)
    vg.dispose()


def test_workspace_grows_and_is_never_above_its_limit():
    vg = engine.VirtualGeometry(max_meshlets=1 << 10)
    mesh = vg.create_mesh(scenes.icosphere_mesh(160), ONE)
    vg.debug_cells_device()
    before = vg.footprint()
    whole = _call(vg, mesh, 3000)  # above the 32 MB that are kept
    assert _bytes(mesh, 3000) > 32 << 20 and vg.footprint() == before
    for n in (1, 2, 3, 500, 7, 1500, 1):
        lo, hi = _call(vg, mesh, n)
        held = vg.footprint() - before
        assert _bytes(mesh, n) <= held <= 32 << 20
    assert lo.shape == (1, mesh.data.meshlet_count)
    # a matrix's bytes do not depend on the call it is in
    assert np.array_equal(lo[0], whole[0][0]) and np.array_equal(hi[0], whole[1][0])
    vg.dispose()
