"""Per-light entries of a vertex's direct light at the counts where the masks of valid entries end (30 shadow
bits, 32 MIS bits).

Under direct lighting every light's part of a sample is independent of the other lights (they share the
draws and the geometry), so the film of all lights is the sum of the films in which one of them emits.
Each film is a rounded sum of at most 2 * 41 terms of both halves per sample; the bound is that many half
units in the last place of the sum of magnitudes, twice over for the two sides."""
import numpy as np
import pytest

from crystal2_gb300 import Context, scenes
from crystal2_gb300 import _native as N

pytestmark = pytest.mark.gpu


def _film(d, lights, emit):
    rng = np.random.default_rng(lights)
    objs = [scenes.disk((0, 0, 0), 8.0, scenes.micro((0.8, 0.7, 0.6), 0.35)), scenes.sphere((0.3, 0.6, 0.2), 0.6, scenes.diffuse((0.5, 0.6, 0.7)))]
    for k in range(lights):
        # large lights, so that BSDF samples reach them
        pos, r, le = (rng.uniform(-3, 3), rng.uniform(1.5, 3.5), rng.uniform(-2, 3)), rng.uniform(0.15, 0.4), rng.uniform(1, 6, 3)
        objs.append(scenes.sphere(pos, r, scenes.diffuse((0, 0, 0)), area_light=le if k in emit else None))
    cfg = scenes.config_json(24, 16, 4, 4, sampler="Default")
    cp, sp = scenes.write_scene(d, cfg, scenes.camera((0, 1.4, -4.5), (0, 0.7, 0), 55), objs)
    with Context(0) as ctx:
        ctx.load(cp, sp, tree=N.TREE_SAH)
        assert ctx.num_lights() == len(emit)
        ctx.set_counting(N.COUNT_TRAVERSAL)  # the level kernels, whatever the wave's size
        p = ctx.render_params()
        p.integrator = N.INTEGRATOR_DIRECT
        ctx.film_clear()
        ctx.render(p)
        return ctx.film()[0].astype(np.float64)


@pytest.mark.parametrize("lights", [2, 29, 30, 31, 32, 33, 40])
def test_lights_add_up(tmp_path, lights):
    every = _film(str(tmp_path), lights, range(lights))
    one = [_film(str(tmp_path), lights, [k]) for k in range(lights)]
    total = np.sum(one, axis=0)
    assert np.mean([f.max() > 0 for f in one]) > 0.9
    assert np.all(np.abs(every - total) <= 4 * 41 * 2.0 ** -23 * np.abs(total) + 1e-30)
