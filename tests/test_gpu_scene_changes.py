"""A context that goes from scene to scene makes the same films as a fresh one: the streams that scenes of more kinds of
material use are made when such a scene first comes, and stay."""
import numpy as np
import pytest

from crystal2_gb300 import Context, scenes
from crystal2_gb300 import _native as N

pytestmark = pytest.mark.gpu

SCENES = {  # buckets with the miss: 3, 11, 5
    "cornell": lambda d: scenes.cornell(d, width=90, height=70, spp=4),
    "material_box": lambda d: scenes.material_box(d, width=101, height=67, spp=4),
    "brdf_box": lambda d: scenes.brdf_box(d, width=80, height=81, spp=4),
}


def _film(ctx, files):
    ctx.load(*files, tree=N.TREE_SAH)
    ctx.film_clear()
    ctx.render(ctx.render_params())
    return ctx.film()[0]


@pytest.mark.parametrize("order", [("cornell", "material_box", "cornell", "brdf_box"), ("brdf_box", "material_box", "brdf_box"), ("material_box", "cornell")])
def test_scene_after_scene(tmp_path, order):
    files = {k: SCENES[k](str(tmp_path / k)) for k in set(order)}
    with Context(0) as ctx:
        for name in order:
            with Context(0) as fresh:
                want = _film(fresh, files[name])
            assert want.max() > 0 and np.array_equal(_film(ctx, files[name]), want)
