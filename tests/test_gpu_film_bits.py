"""A film does not depend on how its paths were grouped: the same bits whether small queues are followed to their end
by one kernel or traced level by level, for every wave size, for a range of samples in one call or in parts, and in
a batch.

The traversal counters switch the finishing kernel off, which makes the level kernels' film."""
import numpy as np
import pytest

from crystal2_gb300 import Batch, Context, scenes
from crystal2_gb300 import _native as N

pytestmark = pytest.mark.gpu

TAIL = N.KERNEL_NAMES.index("tail")


def _box(d, balls, w, h, spp, depth, sampler, accel, lights=0, albedo=0.7):
    """Diffuse box with a quad, a sphere, a disk and a point light (or `lights` sphere lights) and a ball per material."""
    walls = scenes._box_walls(d, -2, 2, 0, 3, -2, 2)
    rng = np.random.default_rng(len(balls) + lights)
    objs = [scenes.mesh(walls[k], scenes.diffuse(albedo * rng.uniform(0.9, 1.0, 3))) for k in sorted(walls)]
    if lights:
        objs += [scenes.sphere((np.cos(k) * 1.5, 2.0 + 0.2 * np.cos(5 * k), np.sin(k) * 1.5), 0.1, scenes.diffuse((0, 0, 0)),
                               area_light=(4 + k % 5, 6, 5)) for k in range(lights)]
    else:
        scenes.quad_obj(d + "/light.obj", [(-0.4, 2.99, -0.4), (-0.4, 2.99, 0.4), (0.4, 2.99, 0.4), (0.4, 2.99, -0.4)], (0, -1, 0))
        objs += [scenes.mesh(d + "/light.obj", scenes.diffuse((0, 0, 0)), area_light=(12, 12, 12)),
                 scenes.sphere((-1.4, 2.3, 1.4), 0.2, scenes.diffuse((0, 0, 0)), area_light=(20, 16, 12)),
                 scenes.disk((-0.5, 2.0, 1.99), 0.3, scenes.diffuse((0, 0, 0)), rotation=(-90, 0, 0), area_light=(6, 6, 9)),
                 scenes.point_light((1.5, 2.5, -1.5), (40, 40, 40))]
    for k, m in enumerate(balls * 2):
        objs.append(scenes.sphere((-1.5 + 0.4 * k, 0.45 + 0.1 * (k % 3), 0.9 - 0.7 * (k % 4)), 0.35, m))
    cfg = scenes.config_json(w, h, spp, depth, accel=accel, sampler=sampler, seed=3)
    return scenes.write_scene(d, cfg, scenes.camera((0, 1.5, -5.5), (0, 1.2, 0), 45), objs, "box")


FAMILIES = {  # at most five kinds of material with the walls'
    "plastic": lambda: [scenes.plastic((0.5, 0.4, 0.3), (0.2, 0.2, 0.2), (0.3, 0.3)), scenes.plastic((0.3, 0.4, 0.6), (0.3, 0.2, 0.1), (0.15, 0.2), ndf="Beckmann"),
                        None, scenes.mirror((0.9, 0.9, 0.9))],
    "glass": lambda: [scenes.micro((0.95, 0.7, 0.4), 0.08, 0.4), scenes.micro((0.9, 0.8, 0.7), 0.3, ndf="Beckmann"), scenes.glass((1, 1, 1), (0.1, 0.1), 1.5),
                      scenes.glass((1, 1, 1), (0.0, 0.0), 1.5)],
    "rough": lambda: [scenes.oren_nayar((0.7, 0.6, 0.7), 0.5), scenes.phong((0.8, 0.8, 0.8), 8), scenes.phong((0.9, 0.7, 0.4), 60), scenes.micro((0.9, 0.9, 0.9), 0.2)],
}


def _make(d, scene, w, h, spp, depth, sampler="Halton", accel="BVH"):
    if scene in FAMILIES:
        return _box(d, FAMILIES[scene](), w, h, spp, depth, sampler, accel)
    if scene == "cornell":
        return scenes.cornell_variant(d, seed=11, width=w, height=h, spp=spp, depth=depth, accel=accel)
    if scene == "yard":
        return scenes.textured_yard(d, width=w, height=h, spp=spp, depth=depth, accel=accel)
    if scene == "many":
        return scenes.many_material(d, n_grid=4, subdiv=2, seed=5, width=w, height=h, spp=spp, depth=depth)
    return scenes.slit_room(d, hf_res=32, width=w, height=h, spp=spp, depth=depth)


def _film(ctx, p, flags=0, parts=1, wave_paths=0):
    ctx.set_counting(flags)
    ctx.film_clear()
    tails = 0
    for k in range(parts):
        q = N.RenderParams.from_buffer_copy(p)
        q.sample_count = p.sample_count // parts
        q.sample_begin = p.sample_begin + k * q.sample_count
        q.wave_paths = wave_paths
        ctx.render(q)
        tails += ctx.stats().kernel_count[TAIL]
    ctx.set_counting(0)
    return ctx.film()[0], tails


# whole waves that the finishing kernel takes at once, and waves whose last levels it takes
@pytest.mark.parametrize("w,h,spp", [(90, 91, 1), (180, 121, 3)])
@pytest.mark.parametrize("integrator", [N.INTEGRATOR_PATH, N.INTEGRATOR_DIRECT])
@pytest.mark.parametrize("scene,sampler,accel", [
    ("plastic", "Halton", "BVH"), ("plastic", "Default", "Brute"), ("glass", "Halton", "Brute"), ("glass", "Stratified", "BVH"), ("rough", "Halton", "BVH"),
    ("rough", "Default", "BVH"), ("cornell", "Halton", "BVH"), ("yard", "Halton", "BVH"), ("many", "Halton", "BVH"), ("slit", "Halton", "Brute"),
])
def test_finishing_kernel_and_levels(tmp_path, scene, sampler, accel, integrator, w, h, spp):
    cp, sp = _make(str(tmp_path), scene, w, h, spp if sampler != "Stratified" else spp and 4, 12, sampler, accel)
    with Context(0) as ctx:
        ctx.load(cp, sp, tree=N.TREE_SAH)
        p = ctx.render_params()
        p.integrator, p.sample_count = integrator, spp
        levels, none = _film(ctx, p, N.COUNT_TRAVERSAL)
        film, tails = _film(ctx, p)
        assert none == 0
        assert tails > 0 or (integrator == N.INTEGRATOR_DIRECT and w * h * spp > 8192)  # a direct wave may end before it is small
        assert levels.max() > 0 and np.array_equal(film, levels)


# lanes of a path: 8 up to 6 lights, 16 up to 14, 32 up to 30; above that the level kernels alone
@pytest.mark.parametrize("lights", [1, 6, 7, 14, 15, 30, 31])
def test_light_counts(tmp_path, lights):
    cp, sp = _box(str(tmp_path), [scenes.micro((0.9, 0.9, 0.9), 0.2), scenes.mirror()], 101, 67, 2, 8, "Halton", "BVH", lights=lights)
    with Context(0) as ctx:
        ctx.load(cp, sp, tree=N.TREE_SAH)
        assert ctx.num_lights() == lights
        p = ctx.render_params()
        levels, _ = _film(ctx, p, N.COUNT_TRAVERSAL)
        film, tails = _film(ctx, p)
        assert (tails > 0) == (lights <= 30)
        assert np.array_equal(film, levels)


@pytest.mark.parametrize("scene", ["cornell", "glass", "many"])
def test_wave_sizes_and_parts(tmp_path, scene):
    cp, sp = _make(str(tmp_path), scene, 160, 121, 8, 12)
    with Context(0) as ctx:
        ctx.load(cp, sp, tree=N.TREE_SAH)
        p = ctx.render_params()
        p.sample_begin = 5
        whole, _ = _film(ctx, p)
        for parts, wave_paths in ((1, 1), (1, 20480 * 3), (2, 0), (8, 0)):
            assert np.array_equal(whole, _film(ctx, p, parts=parts, wave_paths=wave_paths)[0])


# waves above and below what the finishing kernel takes whole, and a room whose paths stay alive
@pytest.mark.parametrize("streams", [0, 2])
@pytest.mark.parametrize("wave_paths", [4096, 1 << 15, 1 << 18])
def test_batch_and_single_renders(tmp_path, streams, wave_paths):
    jobs, want = [], []
    for k, (scene, w, h, spp) in enumerate((("cornell", 160, 121, 16), ("many", 64, 64, 32), ("glass", 200, 150, 4), ("bright", 192, 192, 8))):
        d = tmp_path / str(k)
        d.mkdir()
        cp, sp = (_box(str(d), [scenes.mirror()], w, h, spp, 16, "Halton", "BVH", albedo=0.95) if scene == "bright" else _make(str(d), scene, w, h, spp, 12))
        ctx = Context(0)
        ctx.load(cp, sp, tree=N.TREE_SAH)
        jobs.append((ctx, ctx.render_params()))
        want.append(_film(*jobs[-1])[0])
    b = Batch(0)
    for ctx, p in jobs:
        ctx.film_clear()
        b.add(ctx, p)
    b.tune(wave_paths, streams)
    b.run()
    for (ctx, _), film in zip(jobs, want):
        assert np.array_equal(ctx.film()[0], film)
    b.close()
