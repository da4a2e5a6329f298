"""The visibility pass on index buffers other than vgc_expand's own: the pass caches a meshlet's vertices for the
consecutive triangles that name one draw slot, and must draw every other buffer as the oracle does, bit for bit -
triangles whose indices name several draw slots, indices outside the draw list, a buffer cut off in the middle of a
warp's step, and cuts of a few triangles."""
import numpy as np
import pytest

import oracle as O
from parity_util import Harness, d2h, small_ruins
from vgcut import engine

pytestmark = pytest.mark.gpu

W, H = 333, 187


@pytest.fixture(scope="module")
def scene():
    spec = small_ruins(seed=9, poses=2, quads=0)
    flags = [dict(shadow=True, vertex_data=True) for _ in spec.meshes]
    flags[0]["max_draw_distance"] = 80.0
    return Harness(spec, flags)


def image(h, cam, change, capacity=None, threshold=1.5):
    import torch
    h.gpu(cam, engine.ViewParams(error_threshold=threshold), slot=0)
    cap = h.caps[0]
    idx = torch.zeros(cap, dtype=torch.int32, device="cuda")
    h.vg.expand(0, 0, idx.data_ptr(), cap)
    host = idx.cpu().numpy().view(np.uint32)
    n = int(h.vg.last_stats["requested_indices"][0])
    host[:n] = change(host[:n].copy())
    idx.copy_(torch.from_numpy(host.view(np.int32)))
    cap = n if capacity is None else capacity(n)
    vis = torch.zeros((H, W), dtype=torch.int64, device="cuda")
    h.vg.visibility(0, 0, cam, idx.data_ptr(), cap, vis.data_ptr(), W, H)
    torch.cuda.synchronize()
    out = h.vg.output(0)
    draw_list = d2h(out.draw_list[0], 2 * out.max_drawn * 4).reshape(-1, 4)
    args = d2h(out.draw_args, out.mesh_slots * 2 * 5).reshape(-1, 5)
    maxd = [f.get("max_draw_distance", float("inf")) for f in h.flags]
    want = O.visibility(h.spec.meshes, [True] * len(h.flags), maxd, h.mats, h.inst_slot, host[:cap], draw_list, args,
                        cam, W, H)
    return vis.cpu().numpy().view(np.uint64), want, n


def mixed(idx):
    """Corners swapped with triangles a few places on: within a meshlet, and across two."""
    rng = np.random.default_rng(3)
    at = rng.integers(0, len(idx) - 600, len(idx) // 10)
    to = at + rng.integers(1, 600, len(at))
    idx[at], idx[to] = idx[to], idx[at].copy()
    return idx


def outside(idx):
    rng = np.random.default_rng(4)
    at = rng.integers(0, len(idx), len(idx) // 20)
    idx[at] = rng.integers(0, 1 << 32, len(at), dtype=np.uint64).astype(np.uint32)
    return idx


def alternating(idx):
    """Neighbouring triangles from far apart: every step of a warp names many draw slots."""
    tri = idx.reshape(-1, 3)
    return np.ascontiguousarray(tri[np.random.default_rng(5).permutation(len(tri))]).reshape(-1)


@pytest.mark.parametrize("change", [mixed, outside, alternating])
def test_other_index_buffers(scene, change):
    got, want, _ = image(scene, scene.spec.cameras[0], change)
    assert (got != engine.VIS_EMPTY).any()
    assert np.array_equal(got, want), f"{int((got != want).sum())} pixels differ"


@pytest.mark.parametrize("short", [1, 2, 95, 96, 97])
def test_capacity_inside_a_step(scene, short):
    got, want, n = image(scene, scene.spec.cameras[1], lambda idx: idx, capacity=lambda n: n // 2 - short)
    assert np.array_equal(got, want), f"{int((got != want).sum())} pixels differ"


@pytest.mark.parametrize("threshold", [20.0, 60.0])
def test_few_triangles(scene, threshold):
    got, want, n = image(scene, scene.spec.cameras[0], lambda idx: idx, threshold=threshold)
    assert n > 0
    assert np.array_equal(got, want), f"{int((got != want).sum())} pixels differ"
