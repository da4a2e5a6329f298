"""selectCut of many view-model matrices: the kernel takes them in groups of 8 and the call keeps a workspace up to
32 MB, so a call of any count - around the groups' edges, and one larger than the workspace - must give what the same
matrices give one call each, and calls of growing and shrinking size must not disturb one another."""
import numpy as np
import pytest

from vgcut import engine, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene():
    vg = engine.VirtualGeometry(max_meshlets=4096)
    first = vg.create_mesh(scenes.icosphere_mesh(8, seed=1), np.eye(4, dtype=np.float32).reshape(1, 16))
    mesh = vg.create_mesh(scenes.icosphere_mesh(40, seed=3), np.eye(4, dtype=np.float32).reshape(1, 16))
    yield vg, mesh
    vg.dispose()


def matrices(n):
    rng = np.random.default_rng(n)
    vm = np.zeros((n, 16))
    yaw, s = rng.uniform(0, 2 * np.pi, n), np.exp(0.3 * rng.standard_normal(n))
    vm[:, 0], vm[:, 2], vm[:, 8], vm[:, 10] = np.cos(yaw) * s, -np.sin(yaw) * s, np.sin(yaw) * s, np.cos(yaw) * s
    vm[:, 5], vm[:, 15] = s, 1.0
    vm[:, 14] = -np.exp(rng.uniform(0.5, 4.0, n))
    return vm, s


@pytest.mark.parametrize("n", [33, 1, 7, 8, 9, 16, 17])
@pytest.mark.parametrize("blend", [1.0, 2.0])
def test_groups(scene, n, blend):
    vg, mesh = scene
    vm, s = matrices(n)
    lo, hi = vg.select_cut(mesh.slot, vm, 900.0, 0.1, s, 1.0, blend)
    assert (hi != 0).any()
    for i in range(n):
        l1, h1 = vg.select_cut(mesh.slot, vm[i], 900.0, 0.1, s[i], 1.0, blend)
        assert np.array_equal(lo[i], l1[0]) and np.array_equal(hi[i], h1[0]), f"matrix {i} of {n}"


def test_larger_than_the_kept_workspace(scene):
    vg, mesh = scene
    count = (32 << 20) // (2 * mesh.data.meshlet_count) + 5
    vm, s = matrices(count)
    lo, hi = vg.select_cut(mesh.slot, vm, 900.0, 0.1, s, 1.0, 2.0)
    for a in (0, count // 2, count - 16):
        l1, h1 = vg.select_cut(mesh.slot, vm[a:a + 16], 900.0, 0.1, s[a:a + 16], 1.0, 2.0)
        assert np.array_equal(lo[a:a + 16], l1) and np.array_equal(hi[a:a + 16], h1)
