"""The eight-wide traversal (scenes prepared by the library) against the CPU oracle:
closest hits of every form a scene and a ray can take, bit for bit.

Every other way through the library traces the same rays with the binary trees
(kernel 1, step_policy 1, scenes set as raw buffers), so these cases are the ones that
differ: leaves of one and of many elements, hits at equal distances, transforms far from
the unit, rays that the wide boxes' arithmetic cannot take.
"""
import numpy as np
import pytest

import oracle
from pulse_b200 import _ffi, scenes
from pulse_b200.layout import Instance, Material, Mesh
from pulse_b200.tracer import Context, PulseError, Scene, Target, gbuffer_primary, render_forward

pytestmark = pytest.mark.gpu

MAT = [Material((0.7, 0.7, 0.7, 1), (0, 0, 0, 1), 0.8, 0.5, 0.0)]


def _triangle_mesh(n, seed, size=1.0, spread=0.0):
    rng = np.random.default_rng(seed)
    p = (rng.uniform(-spread, spread, (n, 1, 3)) + rng.normal(size=(n, 3, 3)) * size).reshape(-1, 3)
    return Mesh(p, np.tile([0.0, 1.0, 0.0], (3 * n, 1)), np.zeros((3 * n, 2)), np.arange(3 * n, dtype=np.uint32))


def _spheres(n, level, box, seed=0, scale=lambda rng: 1.0):
    rng = np.random.default_rng(seed)
    mesh = scenes.displaced_icosphere(level, 0.1, seed, radius=1.5)
    inst = [Instance(0, 0, scenes.trs(rng.uniform(-box, box, 3), scenes.random_rotation(rng), scale(rng)))
            for _ in range(n)]
    return [mesh], inst


def _scene(kind):
    """(meshes, instances, BLAS leaf size, TLAS leaf size, half extent the rays start in)"""
    eye = np.eye(4)
    rng = np.random.default_rng(5)
    if kind == "one_triangle":
        return [_triangle_mesh(1, 1)], [Instance(0, 0)], 8, 1, 2.0
    if kind == "one_leaf":
        return [_triangle_mesh(8, 2, spread=2.0)], [Instance(0, 0)], 8, 1, 3.0
    if kind == "nine_triangles":
        return [_triangle_mesh(9, 3, spread=2.0)], [Instance(0, 0), Instance(0, 0, scenes.trs((3, 0, 0)))], 8, 1, 4.0
    if kind.startswith("leaf"):  # leaf sizes within a reference's range and beyond it
        return [_triangle_mesh(600, 4, 0.4, 4.0)], [Instance(0, 0)], int(kind[4:]), 1, 5.0
    if kind == "cornell":
        d = scenes.cornell()
        return d.meshes, d.instances, 4, 1, 1.0
    if kind == "cornell_leaf8":  # instances of several materials in TLAS leaves of up to 4
        d = scenes.cornell()
        return d.meshes, d.instances, 8, 4, 1.0
    if kind == "overlapping":
        return *_spheres(24, 3, 2.0), 8, 1, 3.0
    if kind == "many":  # four levels of the wide instance tree
        return *_spheres(700, 1, 12.0), 4, 1, 12.0
    if kind == "same_centre":  # TLAS leaves that cannot be split
        m = [scenes.displaced_icosphere(2, 0.1, 1)]
        return m, [Instance(0, 0, scenes.trs(scale=(s, s, s))) for s in (1.0, 1.5, 2.0, 2.5)], 8, 1, 3.0
    if kind == "same_centre_many":  # more than a wide node's eight
        m = [scenes.displaced_icosphere(1, 0.1, 1)]
        return m, [Instance(0, 0, scenes.trs(scale=(s, s, s))) for s in np.linspace(1, 3, 20)], 8, 1, 4.0
    if kind == "duplicates":  # every hit at the same distance as another
        m, i = _spheres(4, 2, 2.0)
        m[0].indices = np.concatenate([m[0].indices, m[0].indices])
        return m, i, 3, 1, 3.0
    if kind == "coplanar":  # boxes standing on a floor and against each other
        q = scenes.quad_mesh([(-4, 0, 4), (4, 0, 4), (4, 0, -4), (-4, 0, -4)], (0, 1, 0))
        i = [Instance(0, 0)] + [Instance(1, 0, scenes.trs((x, 0.5, z))) for x in (-1, 0, 1) for z in (-1, 0, 1)]
        return [q, scenes.unit_cube()], i, 4, 1, 2.0
    if kind == "scaled":
        return *_spheres(20, 2, 4.0, 1, lambda r: r.uniform(0.05, 3.0, 3)), 8, 1, 5.0
    if kind == "mirrored_sheared":
        m, i = _spheres(10, 2, 4.0, 2, lambda r: (-1.0, r.uniform(0.3, 2.0), 1.0))
        for k, x in enumerate(i):
            s = eye.copy()
            s[0, 1] = 0.4 * k
            x.object_world = np.asarray(x.object_world) @ s
        return m, i, 8, 1, 5.0
    if kind == "far_away":
        m, i = _spheres(10, 3, 4.0, 3)
        for x in i:
            x.object_world = scenes.trs((2e4, -1e4, 3e4)) @ np.asarray(x.object_world)
        return m, i, 8, 1, 5.0
    if kind == "tiny":
        return *_spheres(10, 2, 0.02, 4, lambda r: 0.01), 8, 1, 0.03
    if kind == "huge":
        return *_spheres(10, 2, 4e3, 5, lambda r: 1e3), 8, 1, 5e3
    if kind == "large_triangles":  # the test's rounding exceeds a small slack
        return [_triangle_mesh(300, 6, 30.0, 60.0), _triangle_mesh(300, 7, 0.3, 40.0)], \
            [Instance(0, 0), Instance(1, 0)], 8, 1, 60.0
    if kind == "singular":  # no inverse: the scene keeps the binary trees
        return *_spheres(6, 2, 2.0, 6, lambda r: (1.0, 0.0, 1.0)), 8, 1, 3.0
    if kind == "projective":
        m, i = _spheres(6, 2, 2.0, 7)
        for x in i:
            x.object_world = np.asarray(x.object_world).copy()
            x.object_world[3] = (0.01, 0.0, 0.02, 1.0)
        return m, i, 8, 1, 3.0
    if kind == "flat_grid":  # boxes without thickness, rays along their planes
        v = scenes.fbm_grid(24, 8.0, 0.0, 1)
        return [v], [Instance(0, 0), Instance(0, 0, scenes.trs((0, 1, 0), scenes.rot_y(rng.uniform())))], 2, 1, 4.0
    raise ValueError(kind)


def _rays(half, centre, seed):
    rng = np.random.default_rng(seed)
    n = 6000
    o = centre + rng.uniform(-1.3, 1.3, (n, 3)) * half
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    d[:900] = np.eye(3)[rng.integers(0, 3, 900)] * rng.choice([-1.0, 1.0], (900, 1))  # along axes
    d[900:1500, 1] = 0.0                                                              # in a plane
    d[900:1500] /= np.maximum(np.linalg.norm(d[900:1500], axis=1, keepdims=True), 1e-3)
    o[1500:2100] = np.round(o[1500:2100] / half * 4) / 4 * half                       # on planes of the scene
    o[2100:2300] += 50.0 * half                                                       # from far away
    d[2100:2300] = centre - o[2100:2300] + rng.normal(size=(200, 3)) * half
    d[2100:2300] /= np.linalg.norm(d[2100:2300], axis=1, keepdims=True)
    d[2300:2400] *= rng.uniform(0.1, 10.0, (100, 1))                                  # not normalized
    d[2400:2420] = 0.0
    d[2420:2430, 0] = np.nan
    o[2430:2440, 1] = np.inf
    o[2440:2450] = 3e9
    return np.concatenate([o, d], 1).astype(np.float32)


KINDS = ["one_triangle", "one_leaf", "nine_triangles", "leaf1", "leaf2", "leaf63", "leaf64", "leaf100", "cornell",
         "cornell_leaf8", "overlapping", "many", "same_centre", "same_centre_many", "duplicates", "coplanar", "scaled",
         "mirrored_sheared", "far_away", "tiny", "huge", "large_triangles", "singular", "projective", "flat_grid"]


@pytest.mark.parametrize("quirks", [1, 0])
@pytest.mark.parametrize("kind", KINDS)
def test_hits_equal_the_oracle(ctx, kind, quirks):
    meshes, instances, leaf, tlas_leaf, half = _scene(kind)
    sb = oracle.assemble(meshes, MAT * 8, instances, 20, leaf, 2, tlas_leaf)
    centre = np.array([2e4, -1e4, 3e4]) if kind == "far_away" else np.zeros(3)
    rays = _rays(half, centre, 11)
    ref = oracle.trace(sb, rays, quirks=quirks)
    sc = Scene(ctx)
    ids = [sc.upload_mesh(m, 20, leaf) for m in meshes]
    sc.set_materials(MAT * 8)
    sc.set_instances(instances, ids, 2, tlas_leaf)
    got = sc.trace(rays, quirks=quirks)
    sc.close()
    assert np.array_equal(got["t"].view(np.uint32), ref["t"].view(np.uint32))
    for a, b in (("instance_index", "instance"), ("triangle_index", "triangle")):
        assert np.array_equal(got[a], ref[b])
    for k in "uv":
        assert np.array_equal(got[k].view(np.uint32), ref[k].view(np.uint32))


@pytest.mark.parametrize("count,box", [(300, 2.0), (3000, 2.0), (3000, 6.0), (20000, 3.0)])
def test_more_children_than_the_stack_takes(ctx, count, box):
    """Instances that overlap many times over: rays enter more boxes of the instance tree
    than its part of the stack takes, from its third level down."""
    meshes, instances = _spheres(count, 1, box, 9, lambda rng: rng.uniform(0.3, 1.0))
    sb = oracle.assemble(meshes, MAT * 8, instances, 20, 4, 2, 1)
    rays = _rays(box, np.zeros(3), 12)
    ref = oracle.trace(sb, rays)
    sc = Scene(ctx)
    ids = [sc.upload_mesh(m, 20, 4) for m in meshes]
    sc.set_materials(MAT * 8)
    sc.set_instances(instances, ids, 2, 1)
    got = sc.trace(rays)
    sc.close()
    assert np.array_equal(got["t"].view(np.uint32), ref["t"].view(np.uint32))
    for a, b in (("instance_index", "instance"), ("triangle_index", "triangle")):
        assert np.array_equal(got[a], ref[b])


@pytest.mark.parametrize("segments", [0, 1, 2, 6, 8, 0xFFFFFFFF])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_frames_equal_the_oracle(ctx, mode, segments):
    """Two accumulated frames of two samples at the default and at every other place of
    the tail kernel: after the first segment, the last but one, the last, never, at once."""
    d = scenes.cornell(67, 41)
    params = dict(max_depth=7, nee_mode=mode, light_pick=1 if mode == 2 else 0, quirks=1, spp=2)
    sb = oracle.assemble(d.meshes, d.materials, d.instances, 20, 4)
    sc = Scene(ctx)
    ids = [sc.upload_mesh(m, 20, 4) for m in d.meshes]
    sc.set_materials(d.materials)
    sc.set_instances(d.instances, ids)
    tg = Target(ctx, d.width, d.height)
    ref = np.zeros((d.height, d.width, 4), np.float32)
    for acc in range(2):
        render_forward(sc, d.view, tg, acc, wf_segments=segments, **params)
        oracle.render(sb, d.view, d.width, d.height, acc, image=ref, **params)
    got = tg.download()
    tg.close()
    sc.close()
    assert np.array_equal(got.view(np.uint32), ref.view(np.uint32))


@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("gap", [0.0, 1e-6, 1e-4, 1e-3, 2e-3, 0.1])
def test_occluder_before_the_light_equals_the_oracle(ctx, mode, gap):
    """A second surface in the light's plane, and within, at and past the slack of a shadow
    ray's limit before it: what hides the light and what does not."""
    d = scenes.cornell(48, 36)
    light = next(x for x in d.instances if max(d.materials[x.material].emissive[:3]) > 0.0)
    dark = next(k for k, m in enumerate(d.materials) if max(m.emissive[:3]) == 0.0)
    half = scenes.trs((0.25, -gap, 0.0))  # over a part of the light, towards the floor
    inst = [*d.instances, Instance(light.mesh, dark, half @ np.asarray(light.object_world))]
    params = dict(max_depth=4, nee_mode=mode, light_pick=0, quirks=0, spp=4)
    sb = oracle.assemble(d.meshes, d.materials, inst, 20, 4)
    sc = Scene(ctx)
    ids = [sc.upload_mesh(m, 20, 4) for m in d.meshes]
    sc.set_materials(d.materials)
    sc.set_instances(inst, ids)
    tg = Target(ctx, d.width, d.height)
    ref = np.zeros((d.height, d.width, 4), np.float32)
    render_forward(sc, d.view, tg, 0, **params)
    oracle.render(sb, d.view, d.width, d.height, 0, image=ref, **params)
    got = tg.download()
    tg.close()
    sc.close()
    assert np.array_equal(got.view(np.uint32), ref.view(np.uint32))


@pytest.mark.parametrize("width", [383, 384])  # of 256 rows: below the line of the dispatch, and on it
@pytest.mark.parametrize("mode", [0, 2])
def test_camera_rays_alone_equal_the_oracle(ctx, mode, width):
    """A frame of one segment over trees of few levels: the wide or the binary trees by its paths."""
    d = scenes.cornell(width, 256)
    params = dict(max_depth=1, nee_mode=mode, light_pick=1 if mode == 2 else 0, quirks=1)
    sb = oracle.assemble(d.meshes, d.materials, d.instances, 20, 4)
    sc = Scene(ctx)
    ids = [sc.upload_mesh(m, 20, 4) for m in d.meshes]
    sc.set_materials(d.materials)
    sc.set_instances(d.instances, ids)
    tg = Target(ctx, width, 256)
    ref = np.zeros((256, width, 4), np.float32)
    render_forward(sc, d.view, tg, 0, **params)
    oracle.render(sb, d.view, width, 256, 0, image=ref, **params)
    got = tg.download()
    # the G-buffer: the same rule
    g = np.asarray(gbuffer_primary(sc, d.view, width, 256))
    want = oracle.gbuffer_primary(sb, d.view, width, 256)
    tg.close()
    sc.close()
    assert np.array_equal(got.view(np.uint32), ref.view(np.uint32))
    assert np.array_equal(g.reshape(-1).view(np.uint32), np.asarray(want).reshape(-1).view(np.uint32))


def _prepare(ctx, meshes, materials, instances, leaf=4):
    sc = Scene(ctx)
    ids = [sc.upload_mesh(m, 20, leaf) for m in meshes]
    sc.set_materials(materials)
    sc.set_instances(instances, ids)
    return sc


@pytest.mark.parametrize("mode", [1, 2])
def test_occluders_whose_boxes_are_rounded_equal_the_oracle(ctx, mode):
    """Small quads between a floor and its light, 40,000 units from the origin: an instance's
    bounds are rounded to 1/256 there, its triangles in object space are not.  A shadow ray that
    passes a quad's edge outside the bounds misses the quad, however far before the light it lies."""
    centre = np.array([2e4, -1e4, 3e4])
    rng = np.random.default_rng(21)

    def at(*p):
        return scenes.trs(centre + p)

    def quad(h, ny):
        return scenes.quad_mesh([(-h, 0, ny * h), (h, 0, ny * h), (h, 0, -ny * h), (-h, 0, -ny * h)], (0, ny, 0))

    meshes = [quad(40.0, 1), quad(8.0, -1), quad(0.77, 1)]
    mats = [Material((0.7, 0.7, 0.7, 1), (0, 0, 0, 1), 0.8, 0.5, 0.0), Material((0.7, 0.7, 0.7, 1), (9, 9, 9, 1), 0.8, 0.5, 0.0)]
    inst = [Instance(0, 0, at(0, 0, 0)), Instance(1, 1, at(0, 70, 0))]
    for x in range(-10, 11):
        for z in range(-10, 11):
            inst.append(Instance(2, 0, at(2.1 * x + rng.uniform(), rng.uniform(2, 20), 2.1 * z + rng.uniform())))
    view = scenes.bevy_view(centre + (3.0, 45.0, 60.0), centre, aspect=96 / 64)
    params = dict(max_depth=3, nee_mode=mode, light_pick=0, quirks=0, spp=4)
    sb = oracle.assemble(meshes, mats, inst, 20, 4)
    sc = _prepare(ctx, meshes, mats, inst)
    tg = Target(ctx, 96, 64)
    ref = np.zeros((64, 96, 4), np.float32)
    render_forward(sc, view, tg, 0, **params)
    oracle.render(sb, view, 96, 64, 0, image=ref, **params)
    got = tg.download()
    tg.close()
    sc.close()
    assert ref[..., :3].max() > 0
    assert np.array_equal(got.view(np.uint32), ref.view(np.uint32))


def test_shadow_ray_past_the_edge_of_the_light_equals_the_oracle(ctx):
    """A texel of the Cornell box with a shadow ray that grazes the light's edge outside its
    bounds: the reference misses the light, and the texel is lit."""
    rng = np.random.default_rng(12)
    d = scenes.cornell()
    mats = [Material((*rng.uniform(0.1, 0.9, 3), 1), m.emissive, rng.uniform(0.2, 1.0), 0.5, 0.0) for m in d.materials]
    view = scenes.bevy_view((rng.uniform(-0.2, 0.2), rng.uniform(-0.2, 0.2), 3.0), (0.0, 0.0, 0.0), aspect=1.0)
    params = dict(max_depth=6, nee_mode=2, light_pick=1, quirks=0, spp=16, seed=12)
    sb = oracle.assemble(d.meshes, mats, d.instances, 20, 8)
    sc = _prepare(ctx, d.meshes, mats, d.instances, 8)
    tg = Target(ctx, 512, 512)
    texels = [106 * 512 + x for x in range(250, 265)]
    ref = np.zeros((512, 512, 4), np.float32)
    render_forward(sc, view, tg, 0, **params)
    oracle.render(sb, view, 512, 512, 0, image=ref, pixels=texels, **params)
    got = tg.download()
    tg.close()
    sc.close()
    a, b = (x.reshape(-1, 4)[texels].view(np.uint32) for x in (got, ref))
    assert np.array_equal(a, b)


def _many_rays(n, half, refused):
    """n rays, of which every second run of `refused` is not for the wide trees."""
    rays = np.resize(_rays(half, np.zeros(3), 13)[:2000], (n, 6))
    rng = np.random.default_rng(14)
    rays[:, :3] += rng.uniform(-0.1, 0.1, (n, 3)) * half
    if refused:
        run = np.arange(n) // refused
        rays[run % 8 == 1, 3:] = 0.0
        rays[run % 8 == 3, 3:] *= 2.5
        rays[run % 8 == 5, 3:] = np.nan
        rays[run % 8 == 7, :3] += 3e9
    return rays.astype(np.float32)


# Warps of a B200's launch: 148 SMs x 4 blocks x 4.  With more than 64 rays for each, pools are
# refilled from the shared cursor.
POOLED = 148 * 16 * 64


@pytest.mark.parametrize("count", [POOLED - 1, POOLED, POOLED + 1, 200003])
@pytest.mark.parametrize("kind,refused", [("cornell", 0), ("cornell", 7), ("cornell", 64), ("cornell", 4096),
                                          ("overlapping", 200), ("duplicates", 0), ("duplicates", 64)])
def test_queries_larger_than_the_pools(ctx, kind, refused, count):
    """Every pool refilled, whole pools of rays to be traced again (refused ones, or hits at
    the same distance), against the binary trees, and some against the oracle."""
    meshes, instances, leaf, tlas_leaf, half = _scene(kind)
    rays = _many_rays(count, half, refused)
    sc = Scene(ctx)
    ids = [sc.upload_mesh(m, 20, leaf) for m in meshes]
    sc.set_materials(MAT * 8)
    sc.set_instances(instances, ids, 2, tlas_leaf)
    want = sc.trace(rays, step_policy=1)
    got = sc.trace(rays)
    sc.close()
    for k in ("instance_index", "triangle_index"):
        assert np.array_equal(got[k], want[k])
    for k in "tuv":
        assert np.array_equal(got[k].view(np.uint32), want[k].view(np.uint32))
    some = np.arange(0, count, 97)
    ref = oracle.trace(oracle.assemble(meshes, MAT * 8, instances, 20, leaf, 2, tlas_leaf), rays[some])
    assert np.array_equal(got["t"][some].view(np.uint32), ref["t"].view(np.uint32))
    assert np.array_equal(got["triangle_index"][some], ref["triangle"])


@pytest.mark.parametrize("mode", [0, 2])
@pytest.mark.parametrize("segments", [0, 0xFFFFFFFF])
def test_frames_of_refused_camera_rays(ctx, mode, segments):
    """A camera beyond the wide trees' range, over more paths than the pools hold."""
    d = scenes.cornell(640, 400)
    view = scenes.bevy_view((0.0, 0.0, 3e9), (0.0, 0.0, 0.0), aspect=1.6)
    params = dict(max_depth=3, nee_mode=mode, light_pick=1 if mode == 2 else 0, wf_segments=segments)
    sc = _prepare(ctx, d.meshes, d.materials, d.instances)
    tg = Target(ctx, 640, 400)
    images = []
    for policy in (1, 0):
        render_forward(sc, view, tg, 0, step_policy=policy, **params)
        images.append(tg.download().copy())
    tg.close()
    sc.close()
    assert np.array_equal(images[0].view(np.uint32), images[1].view(np.uint32))


@pytest.mark.parametrize("count", [1, 6, 40, 8300])  # a root leaf, one block, and the grid's barriers from 8,193 on
@pytest.mark.parametrize("far", ["translation", "extent"])
def test_instance_out_of_range_keeps_the_binary_trees(ctx, count, far):
    """One instance whose bounds pass 1e9 leaves the whole scene to the binary trees; moved
    back, the scene takes the wide ones again."""
    meshes, instances = _spheres(count, 1, 8.0, 15, lambda rng: rng.uniform(0.05, 0.2))
    home = instances[count // 2].object_world
    away = scenes.trs((0, 2e9, 0)) if far == "translation" else scenes.trs((0, 9e8, 0), scale=(2e8, 2e8, 2e8))
    rays = _rays(8.0, np.zeros(3), 16)
    sc = Scene(ctx)
    ids = [sc.upload_mesh(m, 20, 4) for m in meshes]
    sc.set_materials(MAT * 8)
    for world in (away, home):
        instances[count // 2].object_world = world
        sc.set_instances(instances, ids, 2, 1)
        got = sc.trace(rays)
        ref = oracle.trace(oracle.assemble(meshes, MAT * 8, instances, 20, 4, 2, 1), rays)
        assert np.array_equal(got["t"].view(np.uint32), ref["t"].view(np.uint32))
        for a, b in (("instance_index", "instance"), ("triangle_index", "triangle")):
            assert np.array_equal(got[a], ref[b])
    sc.close()


def test_no_memory_for_the_wide_trees():
    """Every allocation of a scene's preparation fails once.  The calls return PULSE_ERR_OOM and
    succeed when repeated, or, where only the wide trees wanted the memory, succeed at once; the
    scene renders the oracle's bits either way."""
    meshes, instances, leaf, _, _ = _scene("coplanar")
    mats = [MAT[0], Material((0.7, 0.7, 0.7, 1), (3.0, 3.0, 3.0, 1), 0.8, 0.5, 0.0)]
    instances[4].material = 1
    view = scenes.bevy_view((1.0, 3.0, 5.0), (0.0, 0.0, 0.0), aspect=1.5)
    params = dict(max_depth=4, nee_mode=2, light_pick=1)
    sb = oracle.assemble(meshes, mats, instances, 20, leaf)
    ref = np.zeros((24, 36, 4), np.float32)
    oracle.render(sb, view, 36, 24, 0, image=ref, **params)

    def prepare(sc):
        ids = [sc.upload_mesh(m, 20, leaf) for m in meshes]
        sc.set_materials(mats)
        sc.set_instances(instances, ids)
        sc.set_instances(instances, ids)  # into the second set of buffers
        sc.update_instances([2], [instances[2].columns()])

    without = refused = 0
    for skip in range(1000):
        with Context(0) as c:  # (its workspaces are not there yet)
            sc = Scene(c)
            c.check(c.lib.pulse_debug_fail_allocations_after(c.h, skip, 1), "arm")
            try:
                try:
                    prepare(sc)
                    failed = False
                except PulseError as e:
                    assert e.code == _ffi.PULSE_ERR_OOM, skip
                    failed = True
                try:
                    Target(c, 8, 8).close()
                except PulseError:
                    break  # the failure was still to come: the preparation allocates no more
            finally:
                c.check(c.lib.pulse_debug_fail_allocations_after(c.h, 0, 0), "disarm")
            if failed:
                refused += 1
                prepare(sc)
            else:
                without += 1
            tg = Target(c, 36, 24)
            render_forward(sc, view, tg, 0, **params)
            assert np.array_equal(tg.download().view(np.uint32), ref.view(np.uint32)), skip
            tg.close()
            sc.close()
    assert refused > 0 and without > 0


def _rays_along(triangles, n, size, seed):
    """Rays that meet a triangle at a small angle, most of them close to an edge."""
    rng = np.random.default_rng(seed)
    t = triangles[rng.integers(0, len(triangles), n)]
    e1 = t[:, 1] - t[:, 0]
    normal = np.cross(e1, t[:, 2] - t[:, 0])
    normal /= np.linalg.norm(normal, axis=1, keepdims=True)
    side = np.cross(normal, e1)
    along = e1 * rng.normal(size=(n, 1)) + side * rng.normal(size=(n, 1))
    along /= np.linalg.norm(along, axis=1, keepdims=True)
    d = along + normal * (rng.choice([-1.0, 1.0], n) * np.exp(rng.uniform(np.log(1e-8), np.log(1e-3), n)))[:, None]
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    b = rng.uniform(size=(n, 3))
    b[: 3 * n // 4, 0] *= np.exp(rng.uniform(np.log(1e-7), 0.0, 3 * n // 4))
    b /= b.sum(1, keepdims=True)
    b = rng.permuted(b, axis=1)
    o = (t * b[:, :, None]).sum(1) - d * (size * np.exp(rng.uniform(np.log(1e-2), np.log(3.0), n)))[:, None]
    return np.concatenate([o, d], 1).astype(np.float32)


@pytest.mark.parametrize("joined", [False, True])
@pytest.mark.parametrize("size,scale", [(200.0, 1.0), (20.0, 1.0), (2.0, 1.0), (0.2, 1000.0)])
def test_rays_along_large_triangles_equal_the_oracle(ctx, size, scale, joined):
    """Triangles of up to hundreds of units: the rounding of a hit's distance is a good part of
    the distance itself, so a hit may lie far before the box that holds it."""
    rng = np.random.default_rng(21)
    p = (rng.uniform(-size, size, (200, 1, 3)) + rng.normal(size=(200, 3, 3)) * size * 0.5).astype(np.float32)
    p = np.concatenate([p, (p[:100, :1] + rng.normal(size=(100, 3, 3)) * size * 0.01)]).astype(np.float32)

    def mesh(q):
        q = q.reshape(-1, 3)
        return Mesh(q, np.tile([0.0, 1.0, 0.0], (len(q), 1)), np.zeros((len(q), 2)), np.arange(len(q), dtype=np.uint32))

    world = scenes.trs(scale=(scale, scale, scale))
    meshes = [mesh(p)] if joined else [mesh(q) for q in p]
    instances = [Instance(k, 0, world) for k in range(len(meshes))]
    rays = _rays_along(p.astype(np.float64) * scale, 150000, size * scale, 22)
    ref = oracle.trace(oracle.assemble(meshes, MAT, instances, 20, 8, 2, 2), rays)
    sc = Scene(ctx)
    ids = [sc.upload_mesh(m, 20, 8) for m in meshes]
    sc.set_materials(MAT)
    sc.set_instances(instances, ids, 2, 2)
    got = sc.trace(rays)
    sc.close()
    assert np.array_equal(got["t"].view(np.uint32), ref["t"].view(np.uint32))
    for a, b in (("instance_index", "instance"), ("triangle_index", "triangle")):
        assert np.array_equal(got[a], ref[b])


@pytest.mark.parametrize("far", [0.0, 1e3])
@pytest.mark.parametrize("axis", [1.0, 0.1, 0.01, 0.001])
def test_sheared_instances_that_coincide_equal_the_oracle(ctx, axis, far):
    """Pairs of instances with the same surface and matrices some roundings apart, squeezed to
    `axis` across their own axes: the distances' roundings grow with the shear."""
    rng = np.random.default_rng(8)
    mesh = scenes.displaced_icosphere(2, 0.1, 1, radius=1.0)
    centre = far * np.array([1.0, 2.0, -3.0])
    instances = []
    for _ in range(8):
        world = (scenes.trs(centre + rng.uniform(-2, 2, 3), scenes.random_rotation(rng))
                 @ np.diag([1.0, axis, rng.uniform(axis, 1.0), 1.0]) @ scenes.trs((0, 0, 0), scenes.random_rotation(rng)))
        other = world.copy()
        other[:3] *= 1.0 + 3e-7 * rng.normal(size=(3, 4))
        instances += [Instance(0, 0, world), Instance(0, 0, other)]
    n = 150000
    o = centre + rng.uniform(-3, 3, (n, 3))
    d = centre + rng.uniform(-2, 2, (n, 3)) - o
    rays = np.concatenate([o, d / np.linalg.norm(d, axis=1, keepdims=True)], 1).astype(np.float32)
    ref = oracle.trace(oracle.assemble([mesh], MAT, instances, 20, 4, 2, 4), rays)
    sc = Scene(ctx)
    ids = [sc.upload_mesh(mesh, 20, 4)]
    sc.set_materials(MAT)
    sc.set_instances(instances, ids, 2, 4)
    got = sc.trace(rays)
    sc.close()
    assert np.array_equal(got["t"].view(np.uint32), ref["t"].view(np.uint32))
    for a, b in (("instance_index", "instance"), ("triangle_index", "triangle")):
        assert np.array_equal(got[a], ref[b])


@pytest.mark.parametrize("copies", [2, 3, 5])
@pytest.mark.parametrize("leaf", [5, 8, 16])
def test_surfaces_modelled_twice_equal_the_oracle(ctx, leaf, copies):
    """Both sides of a surface as triangles of their own, and more copies: hits at the same
    distance, or roundings apart, within one leaf and across the triangles of several steps."""
    mesh = scenes.displaced_icosphere(2, 0.1, 4, radius=1.0)
    one = np.asarray(mesh.indices).reshape(-1, 3)
    turned = [one, one[:, ::-1], one[:, [1, 2, 0]], one, one[:, [2, 1, 0]]][:copies]
    mesh.indices = np.concatenate(turned).reshape(-1).astype(np.uint32)
    rng = np.random.default_rng(3)
    instances = [Instance(0, 0, scenes.trs(rng.uniform(-2, 2, 3), scenes.random_rotation(rng))) for _ in range(6)]
    rays = np.resize(_rays(3.0, np.zeros(3), 17), (30000, 6)).astype(np.float32)
    rays[:, :3] += rng.uniform(-0.5, 0.5, (30000, 3)).astype(np.float32)
    ref = oracle.trace(oracle.assemble([mesh], MAT, instances, 20, leaf, 2, 1), rays)
    sc = Scene(ctx)
    ids = [sc.upload_mesh(mesh, 20, leaf)]
    sc.set_materials(MAT)
    sc.set_instances(instances, ids, 2, 1)
    got = sc.trace(rays)
    sc.close()
    for a, b in (("t", "t"), ("u", "u"), ("v", "v")):
        assert np.array_equal(got[a].view(np.uint32), ref[b].view(np.uint32))
    for a, b in (("instance_index", "instance"), ("triangle_index", "triangle")):
        assert np.array_equal(got[a], ref[b])


@pytest.mark.parametrize("count", [1, 24, 60])  # loose leaves a line: below the rule's limit, about it, and above
def test_many_large_triangles_equal_the_oracle(ctx, count):
    """Instances of a mesh of large triangles, few enough for the wide trees and too many, beside
    small ones: the rule's routes, through two frames of instances that change between them."""
    rng = np.random.default_rng(24)
    big = scenes.displaced_icosphere(2, 0.1, 3, radius=150.0)
    small = scenes.displaced_icosphere(2, 0.1, 5, radius=8.0)
    insts = [Instance(0, 0, scenes.trs(rng.uniform(-200, 200, 3), scenes.random_rotation(rng))) for _ in range(count)]
    insts += [Instance(1, 0, scenes.trs(rng.uniform(-400, 400, 3), scenes.random_rotation(rng))) for _ in range(20)]
    n = 20000
    o = rng.uniform(-500, 500, (n, 3))
    d = rng.uniform(-300, 300, (n, 3)) - o
    rays = np.concatenate([o, d / np.linalg.norm(d, axis=1, keepdims=True)], 1).astype(np.float32)
    sc = Scene(ctx)
    ids = [sc.upload_mesh(m, 20, 8) for m in (big, small)]
    sc.set_materials(MAT)
    for now in (insts, insts[count // 2:], insts):
        sc.set_instances(now, ids)
        got = sc.trace(rays)
        ref = oracle.trace(oracle.assemble([big, small], MAT, now, 20, 8), rays)
        assert np.array_equal(got["t"].view(np.uint32), ref["t"].view(np.uint32))
        for a, b in (("instance_index", "instance"), ("triangle_index", "triangle")):
            assert np.array_equal(got[a], ref[b])
    sc.close()


@pytest.mark.parametrize("leaf", [4, 8])
@pytest.mark.parametrize("turned", [False, True])
def test_margins_grow_after_the_hit(ctx, turned, leaf):
    """Rays onto the edges of a cube, almost along them: a face met by a rounding before the box
    that holds it, the next face's hit within that distance.  Behind the cube's own faces lie the bounds
    of an instance with far larger coordinates, entered after the hit: its margins are not the hit's."""
    rng = np.random.default_rng(25)
    corner = np.array([[0, 0, 0], [0.1, 0, 0], [0, 0.1, 0]])
    p = np.concatenate([corner - 0.49999, 4.9 - corner]) + 1000.0  # two triangles, little in their box
    sparse = Mesh(p, np.tile([0.0, 1.0, 0.0], (6, 1)), np.zeros((6, 2)), np.arange(6, dtype=np.uint32))
    world = scenes.trs((0.1, 0.2, 0.3), scenes.random_rotation(rng)) if turned else np.eye(4)
    instances = [Instance(0, 0, world), Instance(1, 0, world @ scenes.trs((-1000, -1000, -1000)))]
    n = 60000
    axis = rng.integers(0, 3, n)
    rows = np.arange(n)
    target = np.full((n, 3), -0.5)
    target[rows, axis] = rng.uniform(-0.5, 0.5, n)
    d = np.exp(rng.uniform(np.log(1e-3), np.log(0.3), (n, 3)))
    d[rows, axis] = rng.choice([-1.0, 1.0], n)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    o = target - d * np.exp(rng.uniform(np.log(2e-3), np.log(1.0), n))[:, None]
    o, d = o @ world[:3, :3].T + world[:3, 3], d @ world[:3, :3].T
    rays = np.concatenate([o, d], 1).astype(np.float32)
    meshes = [scenes.unit_cube(), sparse]
    ref = oracle.trace(oracle.assemble(meshes, MAT, instances, 20, leaf), rays)
    sc = _prepare(ctx, meshes, MAT, instances, leaf)
    got = sc.trace(rays)
    sc.close()
    assert (ref["t"] < 1e29).sum() > n // 4
    assert np.array_equal(got["t"].view(np.uint32), ref["t"].view(np.uint32))
    for a, b in (("instance_index", "instance"), ("triangle_index", "triangle")):
        assert np.array_equal(got[a], ref[b])
