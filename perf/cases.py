"""The engine's work as its users have it done, through the package's public entry points, over the range it is used in.

A case is a dict of plain values; its ``kind`` says which part of the API it goes through:

* ``frame``: one view per call by the plain launch, the renderer's frame loop. With ``read`` a headless program that
  takes the stats and the draw list to the host; without, a renderer that leaves them in device memory.
* ``batch``: many views of one scene in one CUDA-graph launch, each with this frame's depth image (the HZBs are built
  in the launch) or with its shadow cascades.
* ``budget``: a large world at 4K under a triangle budget, the threshold searched on the device.
* ``serve``: a burst of requests over several resident scenes through the continuous-batching server.
* ``two_pass``: two-pass occlusion, the previous cuts drawn as occluders and this frame's cut against their depth.
* ``visibility``: the closed loop of one view, its cut, index expansion and visibility buffer.
* ``move``: a crowd that moved: new matrices, re-sort along the Morton curve, the next frame's cut.
* ``select``: selectCut for many view-model matrices of one mesh, its fade bytes on the host.
* ``hzb``: the mip chain of one depth image by itself.

Scenes follow the benchmark's ruins-like and large-world workloads (instances at 113,106 per square kilometre, ground
cameras at 2 m), with a mesh library that builds in seconds. The meshes are a program's assets and the same for every
seed; instances, cameras, thresholds, budgets and depth images come from the seed.

A draw list is a set: its order, and with it each entry's place in the index regions, follows atomics and differs from
run to run. A pass therefore returns what does not depend on that order: the counters, the indirect draw arguments, the
HZBs, and images drawn from the list (occluder depth, the depth of the visibility buffer); the ``read`` frames return
the list itself, sorted. Of the counters the words that describe the cut are returned, not those that count how the
engine's passes happened to share the work (words 15..19 and 23). Output capacities are large enough that no list
overflows: which entries an overflowing list keeps follows atomics too.
"""
import math
import os
import sys
from concurrent.futures import ThreadPoolExecutor
from functools import lru_cache

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "three-virtual-geometry_b200"))

from vgcut import build as B  # noqa: E402
from vgcut import engine, scenes  # noqa: E402
from vgcut.camera import Camera, cascade_clips  # noqa: E402

DENSITY = 113_106.0  # instances per square kilometre (the ruins-like scene)
WEIGHT = 4.0  # a mesh is chosen in proportion to triangles^-4: the smallest meshes are placed most, as in that scene
NEAR, FAR = 0.1, 5000.0
LIGHT = (0.35, -1.0, 0.25)
SPLITS = [0.1, 10.0, 40.0, 150.0, 600.0]


def listed():
    return [
        # the smallest call: a viewer of a few objects that reads the cut back each frame (latency, launches, read-back)
        dict(name="frame_small_read", kind="frame", scene="objects", subdivision=64, instances=64, width=1280,
             height=720, threshold=1.0, depth=False, shadow=False, read=True),
        # the small plain scene of the benchmark: one 1M-triangle mesh, 64 instances, 1080p (launch-bound)
        dict(name="frame_objects", kind="frame", scene="objects", subdivision=229, instances=64, width=1920,
             height=1080, threshold=1.0, depth=False, shadow=False, read=False),
        # an ordinary game frame: ruins-like scene, occlusion from this frame's depth, shadow cut along the sun
        dict(name="frame_ruins", kind="frame", scene="ruins", instances=113_106, width=1920, height=1080,
             threshold=1.0, depth=True, shadow=True, read=False),
        # the benchmark's headline: 32 views with their depth images in one graph launch
        dict(name="batch_ruins", kind="batch", instances=113_106, cameras=32, width=1920, height=1080, threshold=1.0,
             depth=True, cascades=0),
        # cameras of mixed size with four shadow cascades each, LOD blend open at 2 px
        dict(name="batch_cascades", kind="batch", instances=113_106, cameras=8, width=2560, height=1440, threshold=2.0,
             depth=False, cascades=4),
        # the large world under a triangle budget
        dict(name="budget_world", kind="budget", instances=1_000_000, cameras=8, width=3840, height=2160,
             budget=6_000_000.0),
        # a serving burst over four scenes
        dict(name="serve_burst", kind="serve", scenes=4, lo=10_000, hi=200_000, requests=128, width=1920, height=1080),
        # two-pass occlusion at the half-resolution depth target, steady state: the occluders are the visible set of the
        # frame before (`first`: the frame after a cut without occlusion, with every hidden meshlet among them)
        dict(name="two_pass", kind="two_pass", instances=113_106, cameras=16, width=960, height=540, first=False),
        # the loop closed: cut, expansion, visibility buffer
        dict(name="visibility_1080p", kind="visibility", instances=113_106, width=1920, height=1080, threshold=1.0),
        # a moving crowd of one mesh
        dict(name="move_crowd", kind="move", instances=50_000, width=1920, height=1080),
        # selectCut for a baker or editor: many placements of the 1M-triangle mesh, blended
        dict(name="select_blend", kind="select", subdivision=229, matrices=64, threshold=1.0, blend=2.0),
        # a depth image of odd size by itself (dynamic resolution): no wide loads, clamped edges
        dict(name="hzb_odd", kind="hzb", width=2555, height=1437),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, top=2560):
    w = _log(rng, 640, top)
    return w, max(1, int(w * rng.choice((9 / 16, 10 / 16, 3 / 4, 9 / 21))))


def draw(rng):
    kind = rng.choice(("frame", "frame", "frame", "batch", "batch", "budget", "serve", "two_pass", "visibility",
                       "move", "select", "hzb"))
    w, h = _size(rng)
    if kind == "frame":
        if rng.random() < 0.5:
            read = rng.random() < 0.5
            return dict(kind=kind, scene="objects", subdivision=_log(rng, 16, 64 if read else 229),
                        instances=_log(rng, 1, 300), width=w, height=h, threshold=round(rng.uniform(0.5, 2.0), 3),
                        depth=False, shadow=False, read=read)
        return dict(kind=kind, scene="ruins", instances=_log(rng, 3_000, 200_000), width=w, height=h,
                    threshold=round(rng.uniform(1.0, 2.5), 3), depth=rng.random() < 0.7, shadow=rng.random() < 0.5,
                    read=False)
    if kind == "batch":
        cascades = rng.choice((0, 0, 2, 4))
        w, h = _size(rng, 1920)
        return dict(kind=kind, instances=_log(rng, 3_000, 113_106), cameras=_log(rng, 2, 8 if cascades else 32),
                    width=w, height=h, threshold=round(rng.uniform(1.0, 2.5), 3), depth=not cascades,
                    cascades=cascades)
    if kind == "budget":
        return dict(kind=kind, instances=_log(rng, 50_000, 1_000_000), cameras=rng.randint(1, 8), width=3840,
                    height=2160, budget=round(rng.uniform(2e6, 8e6)))
    if kind == "serve":
        return dict(kind=kind, scenes=rng.randint(1, 4), lo=3_000, hi=_log(rng, 10_000, 200_000),
                    requests=_log(rng, 8, 128), width=min(w, 1920), height=min(h, 1080))
    if kind == "two_pass":
        return dict(kind=kind, instances=_log(rng, 3_000, 113_106), cameras=rng.randint(1, 16),
                    width=_log(rng, 320, 960), height=_log(rng, 180, 540), first=rng.random() < 0.25)
    if kind == "visibility":
        w, h = _size(rng, 1920)
        return dict(kind=kind, instances=_log(rng, 3_000, 113_106), width=w, height=min(h, 1080),
                    threshold=round(rng.uniform(1.0, 2.5), 3))
    if kind == "move":
        return dict(kind=kind, instances=_log(rng, 200, 50_000), width=w, height=h)
    if kind == "select":
        return dict(kind=kind, subdivision=_log(rng, 16, 229), matrices=_log(rng, 1, 64),
                    threshold=round(rng.uniform(0.5, 2.0), 3), blend=rng.choice((1.0, 2.0)))
    return dict(kind=kind, width=_log(rng, 64, 3840), height=_log(rng, 36, 2160))


# ---------------------------------------------------------------------------------------------------- inputs
@lru_cache(maxsize=None)
def _icosphere(n):
    return scenes.icosphere_mesh(n)


@lru_cache(maxsize=None)
def _library():
    """24 meshes of 50k-800k triangles, log-spaced: displaced icospheres and box lattices by turns."""
    def make(i):
        tris = math.exp(math.log(50_000) + (i + 0.5) / 24 * math.log(16))
        if i % 2 == 0:
            pos, idx = B.gen_icosphere(int(round(math.sqrt(tris / 20))), 1.0 + i * 7 % 24 / 8, 0.07, 2.5, 100 + i)
        else:
            boxes = 4 + i % 12
            pos, idx = B.gen_box_lattice(boxes, int(round(math.sqrt(tris / (12 * boxes)))), 2.0 + i * 7 % 24 / 6, 100 + i)
        return B.build_virtual_mesh(pos, idx, threads=1)

    with ThreadPoolExecutor(max_workers=os.cpu_count()) as ex:
        return list(ex.map(make, range(24)))


def _triangles():
    return [m.stats["leafTriangles"] for m in _library()]


def _extent(n):
    return 1000.0 * math.sqrt(n / DENSITY)


def _ruins(n, seed):
    """n instances of the library's meshes at the ruins density: matrices per mesh."""
    return scenes.serving_scenes(_library(), _triangles(), WEIGHT, seed=seed, count=1, lo=n, hi=n)[0].instances


def _cameras(rng, n, extent, width, height):
    """Ground cameras at 2 m inside the scene, looking along the ground."""
    out = []
    for _ in range(n):
        x, z = rng.uniform(-0.4, 0.4, 2) * extent
        yaw = rng.uniform(0.0, 2 * math.pi)
        out.append(Camera.perspective_look_at((x, 2.0, z), (x + math.cos(yaw), 1.98, z + math.sin(yaw)), 60.0, width,
                                              height, NEAR, FAR))
    return out


def _depth_images(seed, n, width, height):
    """n NDC depth images (n, height, width): 64 screen-aligned quads at 5-500 m over the far plane."""
    rng = np.random.default_rng([seed, 11])
    c, d = -FAR / (FAR - NEAR), -FAR * NEAR / (FAR - NEAR)
    out = torch.ones((n, height, width), device="cuda")
    for image in out:
        for _ in range(64):
            w, h = (0.04 + 0.3 * rng.random()) * width, (0.04 + 0.35 * rng.random()) * height
            x, y = rng.random() * (width - w), rng.random() * (height - h)
            part = image[int(y):int(y + h), int(x):int(x + w)]
            part.clamp_(max=float(d / rng.uniform(5.0, 500.0) - c))
    return out


# ---------------------------------------------------------------------------------------------------- outputs
class _DeviceArray:
    """Device memory of a context as an array; keeps its owner alive."""

    def __init__(self, owner, ptr, shape, kind):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=tuple(shape), typestr=kind, data=(int(ptr), False), version=3,
                                             strides=None)


def _tensor(owner, ptr, shape, kind="<i4"):
    return torch.as_tensor(_DeviceArray(owner, ptr, shape, kind), device="cuda")


def _cut_outputs(vg, first, n):
    """What slots [first, first + n) hold after a cut whatever the order of its draw list: the counters of the cut, its
    per-mesh index regions and its indirect draw arguments."""
    o = vg.output(first)
    c = _tensor(vg, o.counters, (n, engine.COUNTER_HEADER + 8 * o.mesh_slots))
    return dict(counters=c[:, :15], predicted=c[:, 20:23], regions=c[:, engine.COUNTER_HEADER:],
                args=_tensor(vg, o.draw_args, (n, 2 * o.mesh_slots * 2, 5)))


def _mips(vg, slot, first_level):
    info = vg.hzb_info(slot)
    last = info["levels"] - 1
    total = info["offset"][last] + info["width"][last] * info["height"][last]
    start = info["offset"][first_level] if first_level < info["levels"] else total
    return _tensor(vg, info["data"] + 4 * start, (total - start,), "<f4")


class _State:
    """One program's context, what it passes to each call, and the stream it works on."""
    stream = None  # one stream for the whole program, as a renderer has

    def __init__(self, **kw):
        if _State.stream is None:
            _State.stream = torch.cuda.Stream()
        self.sp = _State.stream.cuda_stream
        self.__dict__.update(kw)

    def __del__(self):
        server = self.__dict__.get("server")
        if server is not None:
            server.close()


def _context(**kw):
    options = dict(max_triangles=40_000_000, max_shadow_triangles=40_000_000, max_meshlets=1 << 18)
    options.update(kw)
    return engine.VirtualGeometry(**options)


def _load(vg, instances, **options):
    for data, mats in zip(_library(), instances):
        vg.create_mesh(data, mats, **options)


# ---------------------------------------------------------------------------------------------------- prepare
def _prepare_frame(case, seed):
    rng = np.random.default_rng([seed, 1])
    w, h = case["width"], case["height"]
    p = engine.ViewParams(error_threshold=case["threshold"], fresh_state=True)
    if case["scene"] == "objects":
        vg = _context()
        n = case["instances"]
        side = math.ceil(math.sqrt(n))
        mats = np.zeros((n, 16), np.float32)
        yaw, s = rng.uniform(0, 2 * math.pi, n), np.exp(0.25 * rng.standard_normal(n))
        mats[:, 0], mats[:, 2], mats[:, 8], mats[:, 10] = np.cos(yaw) * s, -np.sin(yaw) * s, np.sin(yaw) * s, np.cos(yaw) * s
        mats[:, 5], mats[:, 15] = s, 1.0
        mats[:, 12] = (np.arange(n) % side - (side - 1) / 2) * 3.0
        mats[:, 14] = (np.arange(n) // side - (side - 1) / 2) * 3.0
        vg.create_mesh(_icosphere(case["subdivision"]), mats)
        half = side * 1.5
        a, d = rng.uniform(0, 2 * math.pi), half * rng.uniform(1.6, 2.6)
        camera = Camera.perspective_look_at((math.cos(a) * d, half * rng.uniform(0.3, 0.8), math.sin(a) * d), (0, 0, 0),
                                            60.0, w, h, NEAR, 1000.0)
        depth = None
    else:
        vg = _context(max_meshlets=1 << 19)
        _load(vg, _ruins(case["instances"], seed), occlusion_culling=case["depth"], cast_shadow=case["shadow"])
        camera = _cameras(rng, 1, _extent(case["instances"]), w, h)[0]
        depth = _depth_images(seed, 1, w, h) if case["depth"] else None
        if case["shadow"]:
            p.shadow_sweep = tuple(60.0 * x for x in LIGHT)
    if depth is not None:
        p.hzb, p.depth_as_mip0 = 0, True
    view = engine.make_view(camera, p, depth=(depth.data_ptr(), w, h) if depth is not None else None)
    vg.params = p
    # a renderer's first frame publishes the scene and lays out the output slots and the HZB
    vg.cut([view])
    torch.cuda.synchronize()
    outs = None if case["read"] else _cut_outputs(vg, 0, 1)
    if depth is not None:
        outs["hzb"] = _mips(vg, 0, 1)
    return _State(vg=vg, view=view, camera=camera, depth=depth, outs=outs, entries=np.zeros(1 << 14, np.uint64))


def _prepare_batch(case, seed):
    rng = np.random.default_rng([seed, 2])
    w, h, n, casc = case["width"], case["height"], case["cameras"], case["cascades"]
    vg = _context(max_meshlets=1 << (20 if casc else 19), output_slots=n * (1 + casc))
    _load(vg, _ruins(case["instances"], seed), occlusion_culling=case["depth"], cast_shadow=casc > 0)
    cameras = _cameras(rng, n, _extent(case["instances"]), w, h)
    depth = _depth_images(seed, n, w, h) if case["depth"] else None
    views = []
    for k, camera in enumerate(cameras):
        p = engine.ViewParams(error_threshold=case["threshold"], state_slot=len(views), hzb=k if case["depth"] else -1,
                              depth_as_mip0=case["depth"])
        views.append(engine.make_view(camera, p, depth=(depth[k].data_ptr(), w, h) if case["depth"] else None))
        for clip in (cascade_clips(camera, LIGHT, SPLITS[:casc + 1]) if casc else ()):
            p = engine.ViewParams(error_threshold=case["threshold"], state_slot=len(views), cascade_clip=clip)
            views.append(engine.make_view(camera, p))
    vg.cut(views, graph=True)  # the first frame publishes the scene and captures the graph
    torch.cuda.synchronize()
    outs = _cut_outputs(vg, 0, len(views))
    if case["depth"]:
        outs["hzb"] = [_mips(vg, k, 1) for k in range(n)]
    return _State(vg=vg, views=views, depth=depth, outs=outs)


def _prepare_budget(case, seed):
    n, extent = case["instances"], 6000.0 * math.sqrt(case["instances"] / 3e6)
    spec = scenes.large_world(_library(), _triangles(), WEIGHT, seed=seed, instances=n, extent=extent,
                              towns=max(1, n // 60_000), town_radius=min(150.0, extent / 8), poses=case["cameras"],
                              width=case["width"], height=case["height"])
    vg = _context(max_meshlets=1 << 20, output_slots=case["cameras"])
    small = set(spec.notes["small_meshes"])
    for i, (data, mats) in enumerate(zip(spec.meshes, spec.instances)):
        vg.create_mesh(data, mats, max_draw_distance=400.0 if i in small else math.inf)
    views = [engine.make_view(c, engine.ViewParams(triangle_budget=case["budget"], threshold_range=(0.5, 24.0),
                                                   state_slot=k, fresh_state=True)) for k, c in enumerate(spec.cameras)]
    vg.cut(views, graph=True)
    torch.cuda.synchronize()
    return _State(vg=vg, views=views, outs=_cut_outputs(vg, 0, len(views)))


def _prepare_serve(case, seed):
    rng = np.random.default_rng([seed, 4])
    w, h = case["width"], case["height"]
    lib = engine.lib()
    resident, depth = [], _depth_images(seed, 8, w, h)
    specs = scenes.serving_scenes(_library(), _triangles(), WEIGHT, seed=seed, count=case["scenes"], lo=case["lo"],
                                  hi=case["hi"])
    state = _State(resident=resident, specs=specs)
    for spec in specs:
        vg = _context(max_meshlets=1 << 19)
        _load(vg, spec.instances, occlusion_culling=True)
        for k in range(len(depth)):
            engine.check(lib.vgc_hzb_build(vg.handle, k, depth[k].data_ptr(), w, h, 1, None))
        resident.append(vg)
    torch.cuda.synchronize()
    state.requests = []
    for _ in range(case["requests"]):
        scene = int(rng.integers(len(specs)))
        camera = _cameras(rng, 1, specs[scene].notes["extent"], w, h)[0]
        p = engine.ViewParams(error_threshold=float(rng.uniform(0.5, 2.0)), hzb=int(rng.integers(len(depth))))
        state.requests.append((scene, engine.make_view(camera, p)))
    state.server = engine.Server(resident, streams=4, max_batch=64, slots_per_scene=case["requests"], linger_us=100)
    state.results = [engine.ServeResult() for _ in state.requests]
    return state


def _prepare_two_pass(case, seed):
    rng = np.random.default_rng([seed, 5])
    w, h, n = case["width"], case["height"], case["cameras"]
    vg = _context(output_slots=2 * n)
    _load(vg, _ruins(case["instances"], seed), occlusion_culling=True, occluder=True)
    before = _cameras(rng, n, _extent(case["instances"]), w, h)
    after = []  # the camera a step later
    for camera in before:
        eye, v = camera.extra["eye"], camera.view
        ahead = np.array([-v[2], -v[6], -v[10]])
        eye = eye + 0.3 * ahead
        after.append(Camera.perspective_look_at(tuple(eye), tuple(eye + ahead), 60.0, w, h, NEAR, FAR))
    depth = torch.empty((n, h, w), device="cuda")
    views, previous = ([engine.make_view(c, engine.ViewParams(state_slot=s + k, hzb=k, depth_as_mip0=True),
                                         depth=(depth[k].data_ptr(), w, h)) for k, c in enumerate(cameras)]
                       for s, cameras in ((n, after), (0, before)))
    images = [d.data_ptr() for d in depth]
    vg.cut([engine.make_view(c, engine.ViewParams(state_slot=k)) for k, c in enumerate(before)])  # the frame before
    if not case["first"]:
        vg.occluder_depth_batch(list(range(n)), before, images, w, h)
        vg.cut(previous)
    torch.cuda.synchronize()
    occluders = engine.OccluderBatch(vg, list(range(n)), after, images)
    outs = _cut_outputs(vg, n, n)
    outs["depth"] = depth
    return _State(vg=vg, views=views, occluders=occluders, outs=outs, case=case)


def _prepare_visibility(case, seed):
    rng = np.random.default_rng([seed, 6])
    w, h = case["width"], case["height"]
    vg = _context(max_meshlets=1 << 19)
    _load(vg, _ruins(case["instances"], seed), vertex_data=True)
    camera = _cameras(rng, 1, _extent(case["instances"]), w, h)[0]
    p = engine.ViewParams(error_threshold=case["threshold"], fresh_state=True)
    view = engine.make_view(camera, p)
    vg.params = p
    vg.cut([view])
    torch.cuda.synchronize()
    vis = torch.empty((h, w), dtype=torch.int64, device="cuda")
    outs = _cut_outputs(vg, 0, 1)
    outs["depth"] = vis.view(torch.int32)[:, 1::2]  # the high words; the low ones name draw slots (the list's order)
    return _State(vg=vg, view=view, camera=camera, vis=vis, outs=outs, case=case,
                  indices=torch.empty(40_000_000 * 3, dtype=torch.int32, device="cuda"))


def _prepare_move(case, seed):
    rng = np.random.default_rng([seed, 7])
    n = case["instances"]
    extent = _extent(n)

    def crowd():
        yaw, s = rng.uniform(0, 2 * math.pi, n), np.exp(0.2 * rng.standard_normal(n))
        m = np.zeros((n, 16), np.float32)
        m[:, 0], m[:, 2], m[:, 8], m[:, 10] = np.cos(yaw) * s, -np.sin(yaw) * s, np.sin(yaw) * s, np.cos(yaw) * s
        m[:, 5], m[:, 15] = s, 1.0
        m[:, 12], m[:, 14] = rng.uniform(-0.5, 0.5, (2, n)) * extent
        return m

    vg = _context()
    mesh = vg.create_mesh(_library()[2], crowd())
    view = engine.make_view(_cameras(rng, 1, extent, case["width"], case["height"])[0],
                            engine.ViewParams(fresh_state=True))
    vg.cut([view])
    torch.cuda.synchronize()
    return _State(vg=vg, mesh=mesh, view=view, moved=crowd(), outs=_cut_outputs(vg, 0, 1))


def _prepare_select(case, seed):
    rng = np.random.default_rng([seed, 8])
    n = case["matrices"]
    vg = _context()
    mesh = vg.create_mesh(_icosphere(case["subdivision"]), np.eye(4, dtype=np.float32).reshape(1, 16))
    vms = np.zeros((n, 16))
    yaw, s = rng.uniform(0, 2 * math.pi, n), np.exp(0.25 * rng.standard_normal(n))
    vms[:, 0], vms[:, 2], vms[:, 8], vms[:, 10] = np.cos(yaw) * s, -np.sin(yaw) * s, np.sin(yaw) * s, np.cos(yaw) * s
    vms[:, 5], vms[:, 15] = s, 1.0
    vms[:, 12:14], vms[:, 14] = rng.uniform(-2, 2, (n, 2)), -np.exp(rng.uniform(math.log(1.5), math.log(60.0), n))
    return _State(vg=vg, mesh=mesh, vms=vms, scale=s, case=case)


def _prepare_hzb(case, seed):
    w, h = case["width"], case["height"]
    vg = _context()
    depth = _depth_images(seed, 1, w, h)
    state = _State(vg=vg, depth=depth, case=case)
    torch.cuda.synchronize()
    engine.check(engine.lib().vgc_hzb_build(vg.handle, 0, depth.data_ptr(), w, h, 1, state.sp))
    torch.cuda.synchronize()
    state.outs = dict(hzb=_mips(vg, 0, 0))
    return state


def prepare(case, seed):
    state = globals()["_prepare_" + case["kind"]](case, seed)
    state.kind = case["kind"] + ("_read" if case.get("read") else "")
    return state


# ---------------------------------------------------------------------------------------------------- run
def _run_frame(s):
    s.vg.cut([s.view], stream=s.sp)
    return s.outs


def _run_frame_read(s):
    s.vg.update(s.camera)
    stats = s.vg.read_stats()
    e = s.vg.draw_list().astype(np.uint64)
    # instance, meshlet, triangle count and blend range; the place in the index regions follows the list's order
    s.entries[:len(e)] = np.sort(e[:, 0] << 44 | e[:, 1] << 24 | e[:, 3])
    s.entries[len(e):] = 0
    return dict(entries=s.entries.view(np.int64), cells=stats["visible_cells"], drawn=np.array(stats["drawn"]),
                indices=np.array(stats["requested_indices"]))


def _run_batch(s):
    s.vg.cut(s.views, stream=s.sp, graph=True)
    return s.outs


_run_budget = _run_batch


def _run_serve(s):
    tickets = [s.server.submit(scene, view) for scene, view in s.requests]
    rows = []
    for ticket, r in zip(tickets, s.results):
        s.server.wait_into(ticket, r)
        s.server.release(ticket)
        t = r.stats
        rows.append((t.visible_cells, t.occluded_instances, t.selected[0], t.drawn[0], t.survived[0], t.work[0],
                     t.requested_indices[0], t.rounds))
    return np.array(rows)


def _run_two_pass(s):
    s.occluders.run(s.case["width"], s.case["height"], stream=s.sp)
    s.vg.cut(s.views, first_slot=len(s.views), stream=s.sp, graph=True)
    return s.outs


def _run_visibility(s):
    s.vg.cut([s.view], stream=s.sp)
    s.vg.expand(0, 0, s.indices.data_ptr(), s.indices.numel(), stream=s.sp)
    s.vg.visibility(0, 0, s.camera, s.indices.data_ptr(), s.indices.numel(), s.vis.data_ptr(), s.case["width"],
                    s.case["height"], stream=s.sp)
    return s.outs


def _run_move(s):
    s.mesh.set_matrices(s.moved)
    s.mesh.commit_instances()
    s.mesh.resort()
    s.vg.cut([s.view], stream=s.sp)
    return dict(s.outs, order=s.mesh.gpu_to_input)


def _run_select(s):
    c = s.case
    return s.vg.select_cut(s.mesh.slot, s.vms, 935.0, NEAR, s.scale, c["threshold"], c["blend"])


def _run_hzb(s):
    c = s.case
    engine.check(engine.lib().vgc_hzb_build(s.vg.handle, 0, s.depth.data_ptr(), c["width"], c["height"], 1, s.sp))
    return s.outs


def run(state):
    return globals()["_run_" + state.kind](state)


# ---------------------------------------------------------------------------------------------------- work, exact
# Sizes that follow from the scenes: bytes of a mesh's test columns per leaf triangle (64 B per meshlet, about 1.7
# meshlets per 100 leaf triangles over all levels), and entries drawn per view in the listed cases' scenes.
_LIBRARY_TRIANGLES = 6_500_000
_BOUNDS = 64 * 0.017
_DRAWN = 80_000


def work(case):
    """Each input read once and each output written once: instances (68 B) and cells, the meshes' bounds, depth images
    and their mips (4/3), drawn entries (16 B); for a raster pass the triangles' vertices and the image."""
    kind = case["kind"]
    px = case.get("width", 0) * case.get("height", 0) * 4
    scene = 68 * case.get("instances", 0) + _LIBRARY_TRIANGLES * _BOUNDS
    mips = px / 3
    if kind == "frame":
        if case["scene"] == "objects":
            tris = 20 * case["subdivision"] ** 2
            return dict(bytes=68 * case["instances"] + tris * _BOUNDS + 16 * 100 * case["instances"], flops=0)
        return dict(bytes=scene + (px + mips if case["depth"] else 0) + 16 * _DRAWN * (1 + case["shadow"]), flops=0)
    if kind == "batch":
        views = case["cameras"] * (1 + case["cascades"])
        return dict(bytes=scene + case["cameras"] * (px + mips if case["depth"] else 0) + 16 * _DRAWN * views, flops=0)
    if kind == "budget":
        return dict(bytes=scene + 16 * _DRAWN * case["cameras"], flops=0)
    if kind == "serve":
        return dict(bytes=case["scenes"] * (68 * math.sqrt(case["lo"] * case["hi"]) + _LIBRARY_TRIANGLES * _BOUNDS) +
                    16 * _DRAWN * case["requests"], flops=0)
    if kind == "two_pass":
        return dict(bytes=scene + case["cameras"] * (2 * px + mips + 2 * 16 * _DRAWN / 8), flops=0)
    if kind == "visibility":
        # drawn entries written and read, 100 triangles each: 4 B of packed triangle and 12 B of indices written, read
        # again, 12 B of position per vertex (half as many as triangles); 8 B per pixel
        return dict(bytes=scene + _DRAWN * 32 + _DRAWN * 100 * (4 + 12 + 12 + 6) + 2 * px, flops=0)
    if kind == "move":
        return dict(bytes=case["instances"] * (64 + 64 + 64 + 8 + 4), flops=0)
    if kind == "select":
        meshlets = 20 * case["subdivision"] ** 2 * 0.017
        return dict(bytes=meshlets * (48 + 2 * case["matrices"]) + case["matrices"] * 152, flops=0)
    return dict(bytes=px * (1 + 4 / 3), flops=0)


def _exact_mips(image, first_level):
    """The max-reduced mip chain in 64 bits: max of 2 x 2, sizes halved rounding up, edges clamped."""
    levels = [image.double()]
    while levels[-1].numel() > 1 and len(levels) < 16:
        a = levels[-1]
        if a.shape[0] % 2 and a.shape[0] > 1:
            a = torch.cat([a, a[-1:]], 0)
        if a.shape[1] % 2 and a.shape[1] > 1:
            a = torch.cat([a, a[:, -1:]], 1)
        a = torch.maximum(a[0::2], a[1::2]) if a.shape[0] > 1 else a
        a = torch.maximum(a[:, 0::2], a[:, 1::2]) if a.shape[1] > 1 else a
        levels.append(a)
    return torch.cat([a.reshape(-1) for a in levels[first_level:]]) if first_level < len(levels) else image[:0, 0].double()


def exact(case, seed):
    """The HZBs; counts, lists and bytes are whole numbers, and a rasterized depth has no value without the rules that
    say which pixels a triangle covers."""
    if case["kind"] == "hzb":
        return dict(hzb=_exact_mips(_depth_images(seed, 1, case["width"], case["height"])[0], 0))
    if case.get("depth"):
        images = _depth_images(seed, case.get("cameras", 1), case["width"], case["height"])
        mips = [_exact_mips(image, 1) for image in images]
        return dict(hzb=mips if case["kind"] == "batch" else mips[0])
    return None
