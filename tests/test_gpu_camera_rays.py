"""Every pixel's paths start, and each once, on films whose last tiles are cut.

The view is filled by one emitter of radiance (4, 2, 1) and a path ends there, so each pixel's sum over n
samples is exactly n times that; a path without a place in the queue, or two in one place, leave a gap."""
import numpy as np
import pytest

from crystal2_gb300 import Context, scenes
from crystal2_gb300 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spp", [1, 5])
@pytest.mark.parametrize("w,h", [(1, 1), (8, 8), (7, 9), (9, 7), (16, 1), (1, 17), (65, 40), (203, 131)])
def test_every_pixel_has_its_paths(tmp_path, w, h, spp):
    objs = [scenes.sphere((0, 0, 0), 100.0, scenes.diffuse((0, 0, 0)), area_light=(4, 2, 1))]
    cfg = scenes.config_json(w, h, spp, 1, sampler="Default", seed=3)
    cp, sp = scenes.write_scene(str(tmp_path), cfg, scenes.camera((0, 0, -110), (0, 0, 0), 2), objs)
    with Context(0) as ctx:
        ctx.load(cp, sp, tree=N.TREE_SAH)
        p = ctx.render_params()
        for flags in (0, N.COUNT_TRAVERSAL):
            ctx.set_counting(flags)
            ctx.film_clear()
            ctx.render(p)
            film, weight = ctx.film()
            assert np.array_equal(weight, np.full_like(weight, spp))
            assert np.array_equal(film, np.broadcast_to(np.float32([4, 2, 1]) * spp, film.shape))
