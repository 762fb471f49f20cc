"""What a user of this library has it do: frames, batches, gradients, the realtime
pass, the per-frame loop, ray queries, tree builds and the upscaling hand-off, over
the sizes of the repository's scenes.

``listed`` are the cases looked at one by one, ``draw`` gives others of the same
ranges, ``prepare`` makes what a program holds before the call (context, scene,
target, inputs), ``run`` is one pass through the public entry points.
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

from pulse_b200 import _ffi, multigpu, scenes, tracer
from pulse_b200.layout import Instance, Material

CORRECTED = dict(nee_mode=2, light_pick=1, quirks=0)   # NEE + MIS, power CDF
REFERENCE = dict(nee_mode=0, light_pick=0, quirks=1)   # the reference's path_trace
DIFFUSE = dict(nee_mode=1, light_pick=0, quirks=1)     # the reference's diffuse NEE estimator
BATCH_SIZES = ((256, 256), (512, 512), (1280, 720), (1920, 1080))
ESTIMATORS = {"corrected": CORRECTED, "reference": REFERENCE, "diffuse": DIFFUSE}


def listed():
    return [
        # Interactive preview of a small scene: one sample per texel, launches and latency count.
        dict(name="cornell_256", kind="frame", scene="cornell", width=256, height=256, spp=1, depth=4,
             estimator="corrected"),
        # Offline quality of the same scene: many samples per call, few triangles.
        dict(name="cornell_512_spp16", kind="frame", scene="cornell", width=512, height=512, spp=16, depth=6,
             estimator="corrected"),
        # The instanced 1080p frame of bench.py: 64 x 327,680 triangles, 8 bounces.
        dict(name="spheres_1080p", kind="frame", scene="spheres", level=7, instances=64, width=1920, height=1080,
             spp=1, depth=8, estimator="corrected"),
        # The reference's own settings (no light sampling, quirks on, 5 bounces) at an odd window size.
        dict(name="spheres_ref_853x481", kind="frame", scene="spheres", level=6, instances=40, width=853, height=481,
             spp=1, depth=5, estimator="reference"),
        # A large outdoor scene: one deep tree, thousands of instances, 16 bounces, 4K.
        dict(name="terrain_4k", kind="frame", scene="terrain", grid=512, instances=4096, width=3840, height=2160,
             spp=1, depth=16, estimator="corrected"),
        # Many small renders in one call.
        dict(name="batch_8", kind="batch", items=8, max_tris=200000, spp=1),
        # Gradients of a material fit.
        dict(name="backward_cornell_256x16", kind="backward", width=256, height=256, samples=16, depth=6),
        # The realtime pass: primary-hit G-buffer, then 2 chained samples of 5 diffuse bounces.
        dict(name="gi_1080p", kind="gi", level=7, instances=64, width=1920, height=1080),
        # The per-frame loop of an application: moving instances, a frame, the image back on the host.
        dict(name="live_720p", kind="live", level=6, instances=64, width=1280, height=720, depth=5),
        # Picking, visibility and baking queries: host rays in, closest hits out.
        dict(name="trace_1000003", kind="trace", scene="spheres", level=6, instances=40, rays=1000003),
        # Acceleration structure of a new mesh.
        dict(name="build_327680", kind="build", level=7, bins=20, leaf=8),
        # The image at the view's resolution, as half floats for the next pass on the device.
        dict(name="resample_1080p_to_4k", kind="resample", width=1920, height=1080, out_width=3840, out_height=2160,
             bilinear=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "frame", "batch", "backward", "gi", "live", "trace", "build",
                       "resample"])
    width = _log(rng, 64, 1920)
    height = max(1, int(width / rng.uniform(1.0, 1.8)))
    if kind == "frame":
        scene = rng.choice(["cornell", "spheres", "terrain"])
        case = dict(kind=kind, scene=scene, width=width, height=height, spp=rng.choice([1, 1, 1, 2, 3]),
                    depth=rng.randint(1, 16), estimator=rng.choice(["corrected", "corrected", "reference", "diffuse"]))
        if scene == "spheres":
            case.update(level=rng.randint(2, 7), instances=_log(rng, 1, 200))
        if scene == "terrain":
            case.update(grid=_log(rng, 8, 512), instances=_log(rng, 1, 4096))
        return case
    if kind == "batch":
        return dict(kind=kind, items=rng.randint(2, 12), max_tris=_log(rng, 20000, 200000), spp=rng.choice([1, 2]))
    if kind == "backward":
        side = _log(rng, 32, 400)
        return dict(kind=kind, width=side, height=max(1, side - rng.randint(0, 31)), samples=rng.randint(1, 16),
                    depth=rng.randint(1, 8))
    if kind == "gi":
        return dict(kind=kind, level=rng.randint(3, 7), instances=_log(rng, 4, 100), width=width, height=height)
    if kind == "live":
        return dict(kind=kind, level=rng.randint(3, 7), instances=_log(rng, 4, 500), width=width, height=height,
                    depth=rng.randint(1, 8))
    if kind == "trace":
        scene = rng.choice(["cornell", "spheres"])
        case = dict(kind=kind, scene=scene, rays=_log(rng, 1000, 1000000))
        if scene == "spheres":
            case.update(level=rng.randint(2, 7), instances=_log(rng, 1, 100))
        return case
    if kind == "build":
        return dict(kind=kind, level=rng.randint(1, 7), bins=rng.choice([2, 8, 16, 20, 32]), leaf=rng.randint(1, 8))
    return dict(kind=kind, width=width, height=height, out_width=_log(rng, 64, 3840), out_height=_log(rng, 64, 2160),
                bilinear=rng.random() < 0.5)


# ------------------------------------------------------------------- scenes
@functools.lru_cache(maxsize=None)
def _icosphere(level):
    return scenes.icosphere(level)  # the same for every seed


def _sphere_mesh(level, seed):
    """scenes.displaced_icosphere at scenes.sphere_radius_for(level), over the kept icosphere."""
    v, f = _icosphere(level)
    r = scenes.sphere_radius_for(level) * (1.0 + 0.1 * scenes.ValueNoise(seed)(v * 3.0))
    v = v * r[:, None]
    return scenes.Mesh(v, scenes.vertex_normals(v, f), np.zeros((v.shape[0], 2)), f.reshape(-1).astype(np.uint32))


def _spheres(level, instances, seed, aspect):
    """scenes.spheres_1080p's layout: instances of one displaced sphere in a box under 8 emissive patches."""
    rng = np.random.default_rng(seed)
    radius = scenes.sphere_radius_for(level)
    box = 10.0 * max(1.0, instances / 64.0) ** (1.0 / 3.0)
    meshes = [_sphere_mesh(level, seed), scenes.disc_mesh(32, 1.5)]
    mats, insts = [], []
    for i in range(instances):
        mats.append(Material((*rng.uniform(0, 1, 3), 1.0), (0, 0, 0, 1), rng.uniform(0.05, 1.0), 0.5,
                             float(rng.random() < 0.3)))
        insts.append(Instance(0, i, scenes.trs(rng.uniform(-box, box, 3), scenes.random_rotation(rng))))
    for j in range(8):
        le = rng.uniform(1.0, 20.0)
        mats.append(Material((0.8, 0.8, 0.8, 1), (le, le, le, 1), 1.0, 0.5, 0.0))
        gx, gz = (j % 4) - 1.5, (j // 4) - 0.5
        insts.append(Instance(1, instances + j, scenes.trs((gx * 5.0, box + 1.5 * radius, gz * 8.0))))
    eye = (rng.uniform(-1, 1), 2.0 + rng.uniform(-0.5, 0.5), 1.8 * box + 3.0 * radius)
    return meshes, mats, insts, scenes.bevy_view(eye, (0.0, 0.0, 0.0), aspect=aspect)


def _cornell(seed, aspect):
    rng = np.random.default_rng(seed)
    d = scenes.cornell()
    mats = [Material((*rng.uniform(0.1, 0.9, 3), 1), m.emissive, rng.uniform(0.2, 1.0), 0.5, 0.0) for m in d.materials]
    view = scenes.bevy_view((rng.uniform(-0.2, 0.2), rng.uniform(-0.2, 0.2), 3.0), (0.0, 0.0, 0.0), aspect=aspect)
    return d.meshes, mats, d.instances, view


def _terrain(grid, instances, seed, aspect):
    rng = np.random.default_rng(seed)
    d = scenes.terrain_scene(n=grid, n_rocks=instances, seed=seed)
    eye = (rng.uniform(-10, 10), 60.0, 220.0)
    return d.meshes, d.materials, d.instances, scenes.bevy_view(eye, (0.0, 0.0, 0.0), aspect=aspect)


def _parts(case, seed):
    aspect = case.get("width", 1) / case.get("height", 1)
    kind = case.get("scene", "spheres")
    if kind == "cornell":
        return _cornell(seed, aspect)
    if kind == "terrain":
        return _terrain(case["grid"], case["instances"], seed, aspect)
    return _spheres(case["level"], case["instances"], seed, aspect)


@functools.lru_cache(maxsize=None)
def _context(pipeline):
    """The program's one context (its frames follow one another), or its context for overlapping frames."""
    ctx = tracer.Context(torch.cuda.current_device())
    ctx.set_pipeline(pipeline)
    return ctx


class _State:
    """What one program holds for a view; its handles are given back with it."""

    def __init__(self, case):
        self.case, self.frame, self.handles = case, 0, []
        self.ctx = _context(2 if case["kind"] == "live" else 1)

    def scene(self, meshes, mats, insts, bins=20, leaf=8):
        s = tracer.Scene(self.ctx)
        self.handles.append(s)
        ids = [s.upload_mesh(m, bins, leaf) for m in meshes]
        s.set_materials(mats)
        s.set_instances(insts, ids)
        return s, ids

    def target(self, width, height):
        t = tracer.Target(self.ctx, width, height)
        self.handles.append(t)
        return t

    def __del__(self):
        try:
            self.ctx.sync()
            for h in self.handles:
                h.close()
        except Exception:  # the interpreter or the library is going down
            pass


def prepare(case, seed):
    st = _State(case)
    kind = case["kind"]
    rng = np.random.default_rng(seed + 77)
    if kind == "frame":
        meshes, mats, insts, st.view = _parts(case, seed)
        st.s, _ = st.scene(meshes, mats, insts)
        st.t = st.target(case["width"], case["height"])
        st.params = dict(ESTIMATORS[case["estimator"]], max_depth=case["depth"], spp=case["spp"], seed=seed & 0xffff)
    elif kind == "batch":
        st.items = []
        for k in range(case["items"]):
            size = BATCH_SIZES[k % len(BATCH_SIZES)]
            d, = scenes.batch_scenes(seed + k, 1, 1e4, case["max_tris"], (size,))
            s, _ = st.scene(d.meshes, d.materials, d.instances)
            st.items.append(tracer.BatchItem(s, d.view, st.target(*size), 0, 1 + 3 * k % 8, k))
        st.params = dict(CORRECTED, spp=case["spp"])
    elif kind == "backward":
        w, h = case["width"], case["height"]
        meshes, mats, insts, st.view = _cornell(seed, w / h)
        st.s, _ = st.scene(meshes, mats, insts)
        g = np.zeros((h, w, 4), np.float32)
        g[..., :3] = (1.0 + 0.3 * rng.normal(size=(h, w, 3))) * (2.0 / (3.0 * w * h))
        st.dimage = g
        st.params = dict(CORRECTED, max_depth=case["depth"], seed=seed & 0xffff)
    elif kind == "gi":
        w, h = case["width"], case["height"]
        meshes, mats, insts, st.view = _parts(case, seed)
        st.s, _ = st.scene(meshes, mats, insts)
        st.t = st.target(w, h)
        st.gbuffer = torch.empty((h, w, 16), dtype=torch.float32, device="cuda")
        st.params = dict(seed=seed & 0xffff)
    elif kind == "live":
        w, h = case["width"], case["height"]
        meshes, mats, insts, view = _parts(case, seed)
        st.s, ids = st.scene(meshes, mats, insts)
        st.t = st.target(w, h)
        st.view = tracer.make_view(view)
        st.n = len(insts)
        st.descs = (_ffi.InstanceDesc * st.n)()
        for d, i in zip(st.descs, insts):
            d.object_world[:] = [float(x) for x in i.columns()]
            d.mesh_id, d.material_index = ids[i.mesh], i.material
        words = np.frombuffer(st.descs, np.float32).reshape(st.n, -1)
        st.heights = words[:case["instances"], 13]  # the spheres' y translations
        st.speeds = rng.uniform(-0.2, 0.2, case["instances"]).astype(np.float32)
        st.bvh = _ffi.BvhParams(2, 1)
        st.p = tracer.render_params(**CORRECTED, max_depth=case["depth"], seed=seed & 0xffff)
        st.images = [torch.zeros((h, w, 4), dtype=torch.float32).pin_memory() for _ in range(2)]
    elif kind == "trace":
        meshes, mats, insts, view = _parts(case, seed)
        st.s, _ = st.scene(meshes, mats, insts)
        st.rays = torch.from_numpy(_rays(case, view, rng)).pin_memory()
        st.hits = torch.zeros((case["rays"], 5), dtype=torch.float32).pin_memory()  # _ffi.HIT_DTYPE rows
        st.p = tracer.render_params()
    elif kind == "build":
        mesh = _sphere_mesh(case["level"], seed)
        n = mesh.triangle_count
        st.prims = torch.zeros((n, 12), dtype=torch.float32).pin_memory()
        for k in range(3):
            st.prims.numpy()[:, 4 * k:4 * k + 3] = mesh.positions[mesh.indices[k::3]]
        st.nodes = torch.zeros((2 * n - 1, 8), dtype=torch.int32).pin_memory()
        st.indices, st.count = torch.zeros(n, dtype=torch.int32).pin_memory(), C.c_uint32(0)
        st.bvh = _ffi.BvhParams(case["bins"], case["leaf"])
    else:
        st.t = st.target(case["width"], case["height"])
        st.t.upload(_image(case, seed))
        st.out = torch.empty((case["out_height"], case["out_width"], 4), dtype=torch.float16, device="cuda")
    return st


def _rays(case, view, rng):
    """Rays from around the eye toward points around the scene's middle."""
    n = case["rays"]
    spread = 1.0 if case["scene"] == "cornell" else 12.0
    o = view.world_position + rng.normal(size=(n, 3)) * 0.02 * spread
    d = rng.uniform(-spread, spread, (n, 3)) - o
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return np.concatenate([o, d], 1).astype(np.float32)


def _image(case, seed):
    """A rendered image's range of values: mostly dim, few bright texels."""
    g = np.random.default_rng(seed)
    img = np.exp(g.normal(-2.0, 1.5, (case["height"], case["width"], 4))).astype(np.float32)
    img[..., 3] = 1.0
    return img


def _image_of(st, target):
    view = multigpu.target_view(target)
    view.owner = st  # the image is the target's memory: the view keeps its owner
    return view


def run(st):
    kind = st.case["kind"]
    if kind == "frame":
        tracer.render_forward(st.s, st.view, st.t, st.frame, **st.params)
        st.frame += 1
        return _image_of(st, st.t)
    if kind == "batch":
        for it in st.items:
            it.accumulation_count = st.frame
        st.frame += 1
        tracer.render_batch(st.ctx, st.items, **st.params)
        return [_image_of(st, it.target) for it in st.items]
    if kind == "backward":
        return tracer.render_backward(st.s, st.view, st.case["width"], st.case["height"], st.case["samples"],
                                      st.dimage, **st.params)
    if kind == "gi":
        tracer.gbuffer_primary(st.s, st.view, st.case["width"], st.case["height"], out=st.gbuffer)
        tracer.render_gi(st.s, st.gbuffer, st.t, st.case["width"], st.case["height"], **st.params)
        return [st.gbuffer, _image_of(st, st.t)]
    if kind == "live":
        lib, image = st.ctx.lib, st.images[st.frame % 2]
        st.heights += st.speeds if st.frame % 8 < 4 else -st.speeds
        st.ctx.check(lib.pulse_instances_set(st.s.h, st.descs, st.n, C.byref(st.bvh)), "instances")
        st.ctx.check(lib.pulse_render_forward(st.s.h, C.byref(st.view), st.t.h, 0, C.byref(st.p)), "render")
        if st.frame:
            st.ctx.check(lib.pulse_target_download_wait(st.t.h), "wait for the previous frame's copy")
        st.ctx.check(lib.pulse_target_download_async(st.t.h, C.c_void_p(image.data_ptr())), "copy")
        st.frame += 1
        return image  # complete once the device is idle
    if kind == "trace":
        st.ctx.check(st.ctx.lib.pulse_trace(st.s.h, C.c_void_p(st.rays.data_ptr()), st.case["rays"], C.byref(st.p),
                                            C.c_void_p(st.hits.data_ptr())), "trace")
        ids = st.hits.view(torch.int32)
        return {"t": st.hits[:, 0], "instance_index": ids[:, 1], "triangle_index": ids[:, 2], "u": st.hits[:, 3],
                "v": st.hits[:, 4]}
    if kind == "build":
        ptr = [C.c_void_p(a.data_ptr()) for a in (st.prims, st.nodes, st.indices)]
        st.ctx.check(st.ctx.lib.pulse_build_blas(st.ctx.h, ptr[0], st.prims.shape[0], C.byref(st.bvh), ptr[1],
                                                 C.byref(st.count), ptr[2]), "build")
        return [st.nodes, st.indices, st.count.value]
    st.ctx.check(st.ctx.lib.pulse_target_resample(st.t.h, st.case["out_width"], st.case["out_height"],
                                                  int(st.case["bilinear"]), C.c_void_p(st.out.data_ptr()), 0), "resample")
    multigpu.after_library(st.ctx)
    return st.out


# --------------------------------------------------------------------- work
def _triangles(case):
    """(stored triangles, triangles of one entered mesh, instances)."""
    if case.get("scene") == "cornell" or case["kind"] == "backward":
        return 26, 12, 8
    if case.get("scene") == "terrain":
        return 2 * (case["grid"] - 1) ** 2 + 20480 + 200, 2 * (case["grid"] - 1) ** 2, case["instances"] + 51
    return 20 * 4 ** case["level"] + 32, 20 * 4 ** case["level"], case["instances"] + 8


BYTES_PER_TRIANGLE = 48 + 80 + 4 + 32  # position, attributes, index, its share of the tree
BOX, TRIANGLE, SHADING = 20, 45, 300   # operations of a box test, a triangle test, a shaded hit


def _ray_flops(tris, instances):
    """One descent to a leaf of the instance tree and of one mesh tree, both children tested at each level."""
    return (math.log2(instances + 1) + math.log2(tris + 1)) * 2 * BOX + 2 * TRIANGLE


def work(case):
    kind = case["kind"]
    if kind == "build":
        n = 20 * 4 ** case["level"]
        # read the triangles, write nodes (about n / leaf) and indices; every level bins every centroid
        return {"bytes": n * (48 + 4) + 64 * n / case["leaf"], "flops": n * math.log2(n / case["leaf"] + 2) * 3 * 8}
    if kind == "resample":
        src, dst = case["width"] * case["height"], case["out_width"] * case["out_height"]
        return {"bytes": 16 * min(src, dst * 4) + 8 * dst, "flops": dst * (40 if case["bilinear"] else 8)}
    if kind == "batch":
        # mean of the four resolutions, about 2 bounces of two rays
        paths = case["items"] * 861184 * case["spp"]
        tris = math.sqrt(1e4 * case["max_tris"])
        return {"bytes": case["items"] * tris * BYTES_PER_TRIANGLE + 16 * paths,
                "flops": paths * 4 * (_ray_flops(tris, 3) + SHADING)}
    stored, tris, instances = _triangles(case)
    scene_bytes = stored * BYTES_PER_TRIANGLE + instances * 200
    per_ray = _ray_flops(tris, instances)
    if kind == "trace":
        return {"bytes": stored * (48 + 32) + case["rays"] * (24 + 20), "flops": case["rays"] * per_ray}
    texels = case["width"] * case["height"]
    if kind == "gi":
        # the primary ray, then per sample about 2 bounces of two rays
        return {"bytes": scene_bytes + texels * (64 + 64 + 16), "flops": texels * (1 + 2 * 4) * (per_ray + SHADING / 2)}
    paths = texels * case.get("spp", case.get("samples", 1))
    bounces = min(case["depth"], 2.5)  # roulette and misses end most paths early
    rays = bounces * (1 if case.get("estimator") == "reference" else 2)
    flops = paths * (rays * per_ray + bounces * SHADING)
    if kind == "backward":
        return {"bytes": scene_bytes + 16 * texels, "flops": 2 * flops}
    return {"bytes": scene_bytes + 16 * texels * (2 if kind == "frame" else 1), "flops": flops}


# -------------------------------------------------------------------- exact
def exact(case, seed):
    """64-bit values where the outputs have such: the resampled image, and the hits of rays over few triangles.

    Rendered images and their gradients have none: every path takes discrete
    decisions (lobe, roulette, light) that depend on the 32-bit random stream
    and rounding, so a 64-bit run follows other paths."""
    if case["kind"] == "resample":
        return _exact_resample(case, seed)
    if case["kind"] == "trace" and case["scene"] == "cornell" and case["rays"] <= 1000000:
        return _exact_trace(case, seed)
    return None


def _exact_resample(case, seed):
    img = torch.from_numpy(_image(case, seed)).cuda().double()
    h, w = img.shape[:2]
    ow, oh = case["out_width"], case["out_height"]

    def axis(n_out, n_in):
        # the sampling position itself is 32-bit in the definition: (k + 0.5) / n_out * n_in
        k = torch.arange(n_out, device="cuda", dtype=torch.float32)
        return (k + 0.5) / torch.tensor(float(n_out), device="cuda") * float(n_in)

    px, py = axis(ow, w), axis(oh, h)
    if not case["bilinear"]:
        return img[py.floor().long().clamp(max=h - 1)][:, px.floor().long().clamp(max=w - 1)].cpu().numpy()
    px, py = px - 0.5, py - 0.5
    fx, fy = (px - px.floor()).double()[None, :, None], (py - py.floor()).double()[:, None, None]
    x0, y0 = px.floor().long(), py.floor().long()
    rows = img[y0.clamp(0, h - 1)] * (1 - fy) + img[(y0 + 1).clamp(0, h - 1)] * fy
    out = rows[:, x0.clamp(0, w - 1)] * (1 - fx) + rows[:, (x0 + 1).clamp(0, w - 1)] * fx
    return out.cpu().numpy()


def _exact_trace(case, seed):
    meshes, _, insts, view = _parts(case, seed)
    rays = _rays(case, view, np.random.default_rng(seed + 77))
    o = torch.from_numpy(rays[:, :3]).cuda().double()
    d = torch.from_numpy(rays[:, 3:]).cuda().double()
    best = torch.full((o.shape[0],), 1e30, dtype=torch.float64, device="cuda")
    bu, bv = torch.zeros_like(best), torch.zeros_like(best)
    for inst in insts:
        m = meshes[inst.mesh]
        ow = torch.from_numpy(np.asarray(inst.object_world, np.float32)).cuda().double()
        wo = torch.linalg.inv(ow)
        lo, ld = o @ wo[:3, :3].T + wo[:3, 3], d @ wo[:3, :3].T
        scale = ld.norm(dim=1)
        ld = ld / scale[:, None]
        p = torch.from_numpy(m.positions[m.indices].reshape(-1, 3, 3)).cuda().double()
        for tri in p:
            e1, e2 = tri[1] - tri[0], tri[2] - tri[0]
            hh = torch.linalg.cross(ld, e2.expand_as(ld))
            a = hh @ e1
            s = lo - tri[0]
            u = (s * hh).sum(1) / a
            q = torch.linalg.cross(s, e1.expand_as(s))
            v, t = (ld * q).sum(1) / a, (q @ e2) / a
            world = t / scale
            ok = (a.abs() >= 1e-4) & (u >= 0) & (v >= 0) & (u + v <= 1) & (t > 0.001) & (world < best)
            best, bu, bv = torch.where(ok, world, best), torch.where(ok, u, bu), torch.where(ok, v, bv)
    return {"t": best.cpu().numpy(), "instance_index": None, "triangle_index": None, "u": bu.cpu().numpy(),
            "v": bv.cpu().numpy()}
