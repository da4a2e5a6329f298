"""Instance updates and re-sorts of a resident scene leave the host mirror behind; a mesh added afterwards re-uploads it
whole. Whatever order moves, re-sorts, added meshes and reads come in, the device's instances and cells must be those of
the matrices the caller set, in the order the calls reported."""
from types import SimpleNamespace

import numpy as np
import pytest

from parity_util import Harness, grid_matrices
from test_gpu_edges import camera_at
from vgcut import engine, scenes

pytestmark = pytest.mark.gpu


def expected(h, matrices):
    return np.concatenate([m[mesh.gpu_to_input] for mesh, m in zip(h.vg.meshes, matrices)])


@pytest.mark.parametrize("n", [1, 127, 128, 129, 700])
@pytest.mark.parametrize("read_between", [False, True])
def test_moves_resorts_and_added_meshes(n, read_between):
    data = scenes.icosphere_mesh(8, seed=4)
    rng = np.random.default_rng(n)
    mats = [grid_matrices(n, 3.0, 1), grid_matrices(257, 2.0, 2)]
    h = Harness(SimpleNamespace(meshes=[data, data], instances=[m.copy() for m in mats]), [{}, {}])
    view = engine.make_view(camera_at((-10.0, 12.0, -10.0), (20.0, 0.0, 20.0)))
    h.vg.cut([view])  # resident

    def move(k, some):
        mesh, m = h.vg.meshes[k], mats[k]
        at = rng.choice(len(m), max(1, len(m) // some), replace=False)
        for i in at:
            m[i, 12:15] += rng.uniform(-40, 40, 3).astype(np.float32)
            mesh.set_matrix_at(int(i), m[i])
        mesh.commit_instances()

    def check():
        dev = h.vg.debug_cells_device()  # publishes a pending upload
        host, inst = h.vg.debug_scene()
        assert np.array_equal(inst, expected(h, mats)), "instances"
        assert np.array_equal(dev.view(np.uint32), host.view(np.uint32)), "device cells against the host's computation"

    move(0, 3)
    h.vg.meshes[0].resort()
    if read_between:
        check()
    move(0, 2)
    move(1, 5)
    mats.append(grid_matrices(70, 5.0, 3))
    h.vg.create_mesh(data, mats[2])  # the pending upload carries the mirror
    move(0, 4)                       # before it is published
    h.vg.meshes[1].resort()
    move(1, 1)
    check()
    mats[0][:, 13] += 2.0
    h.vg.meshes[0].set_matrices(mats[0])
    h.vg.meshes[0].commit_instances()
    h.vg.meshes[0].resort()
    check()
    h.vg.dispose()
