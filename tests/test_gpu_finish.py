"""Small queues followed to their end by one kernel against the level-by-level kernels.

The traversal counters switch the finishing kernel off, so the same render runs both ways.  Both use the
same samples, surfaces and directions; sums of radiance may be contracted differently, some 2^-23 of a
sample's radiance per vertex (at most 16 here), and one such bit in a direction could turn a path."""
import numpy as np
import pytest

from crystal2_gb300 import Context, scenes
from crystal2_gb300 import _native as N

pytestmark = pytest.mark.gpu

SCENES = {
    "cornell": lambda d, **k: scenes.cornell_variant(d, seed=11, **k),
    "brdf_box": scenes.brdf_box,
    "textured_yard": scenes.textured_yard,
    "many": lambda d, **k: scenes.many_material(d, n_grid=4, subdiv=2, seed=5, **k),
    "slit": lambda d, **k: scenes.slit_room(d, hf_res=32, **k),
}


def _film(ctx, p, flags):
    ctx.set_counting(flags)
    ctx.film_clear()
    ctx.render(p)
    return ctx.film()


def _same(ctx, p):
    ref, w0 = _film(ctx, p, N.COUNT_TRAVERSAL)
    got, w1 = _film(ctx, p, 0)
    again, _ = _film(ctx, p, 0)
    assert np.array_equal(w0, w1)
    assert np.array_equal(got, again)
    scale = np.maximum(np.abs(ref), np.sqrt(np.mean(ref.astype(np.float64) ** 2)))
    off = np.max(np.abs(got - ref) / scale, axis=-1)
    assert np.mean(off > 16 * 2.0 ** -23 * 8) <= 1e-3
    return ref


# whole waves at most as large as the kernel's limit (one path, one warp, odd frames), and larger waves whose
# late levels come down to it; 8 lights take 16 lanes a path
@pytest.mark.parametrize("scene,w,h,spp,depth", [
    ("cornell", 1, 1, 1, 8), ("cornell", 13, 7, 1, 8), ("cornell", 64, 64, 2, 1), ("brdf_box", 90, 91, 1, 6),
    ("textured_yard", 75, 50, 2, 6), ("many", 101, 67, 1, 16), ("many", 160, 121, 4, 16), ("slit", 120, 81, 4, 12), ("cornell", 201, 99, 4, 8),
])
@pytest.mark.parametrize("integrator", [N.INTEGRATOR_PATH, N.INTEGRATOR_DIRECT])
def test_finish_matches_levels(tmp_path, scene, w, h, spp, depth, integrator):
    cp, sp = SCENES[scene](str(tmp_path), width=w, height=h, spp=spp, depth=depth)
    with Context(0) as ctx:
        ctx.load(cp, sp, tree=N.TREE_SAH)
        p = ctx.render_params()
        p.integrator = integrator
        p.sample_begin = 3
        _same(ctx, p)


def test_many_lights(tmp_path):
    d = str(tmp_path)
    objs = [scenes.sphere((0, -100, 0), 100.0, scenes.diffuse((0.6, 0.6, 0.6))), scenes.sphere((0, 0.5, 0), 0.5, scenes.mirror())]
    objs += [scenes.sphere((np.cos(k) * 2, 1.5, np.sin(k) * 2), 0.1, scenes.diffuse((0, 0, 0)), area_light=(4 + k, 6, 5)) for k in range(11)]
    objs.append(scenes.point_light((0, 3, 0), (20, 20, 20)))
    cfg = scenes.config_json(64, 40, 2, 6, sampler="Default", seed=3)
    cp, sp = scenes.write_scene(d, cfg, scenes.camera((0, 1.5, -4), (0, 0.5, 0), 50), objs)
    with Context(0) as ctx:
        ctx.load(cp, sp, tree=N.TREE_SAH)
        assert ctx.num_lights() == 12
        assert _same(ctx, ctx.render_params()).mean() > 0.01
