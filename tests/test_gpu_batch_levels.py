"""Captured waves follow their own queue: they hand over to the finishing kernel when few paths are left, not
after a number of levels that suits some scene."""
import time

import numpy as np
import pytest

from crystal2_gb300 import Batch, Context, scenes
from crystal2_gb300 import _native as N

pytestmark = pytest.mark.gpu


def _room(d, albedo, side, spp, depth):
    """A closed room of one albedo, lit by a quad."""
    walls = scenes._box_walls(d, -2, 2, 0, 3, -2, 2)
    scenes.quad_obj(d + "/front.obj", [(-2, 0, -2), (-2, 3, -2), (2, 3, -2), (2, 0, -2)], (0, 0, 1))
    scenes.quad_obj(d + "/light.obj", [(-0.4, 2.99, -0.4), (-0.4, 2.99, 0.4), (0.4, 2.99, 0.4), (0.4, 2.99, -0.4)], (0, -1, 0))
    objs = [scenes.mesh(walls[k], scenes.diffuse((albedo,) * 3)) for k in sorted(walls)] + [scenes.mesh(d + "/front.obj", scenes.diffuse((albedo,) * 3))]
    objs += [scenes.mesh(d + "/light.obj", scenes.diffuse((0, 0, 0)), area_light=(12, 12, 12)), scenes.sphere((0.5, 0.6, 0.3), 0.6, scenes.mirror())]
    cfg = scenes.config_json(side, side, spp, depth)
    return scenes.write_scene(d, cfg, scenes.camera((0, 1.5, -1.9), (0, 1.2, 0), 70), objs, "room")


def _jobs(tmp_path, n, *args):
    jobs = []
    for k in range(n):
        d = tmp_path / str(k)
        d.mkdir()
        cp, sp = _room(str(d), *args)
        ctx = Context(0)
        ctx.load(cp, sp, tree=N.TREE_SAH)
        jobs.append((ctx, ctx.render_params()))
    return jobs


# depths around the levels before the loop and an odd number of levels in it
@pytest.mark.parametrize("depth", [1, 2, 3, 4, 5, 16])
@pytest.mark.parametrize("streams", [0, 1])
def test_depths(tmp_path, depth, streams):
    [(ctx, p)] = _jobs(tmp_path, 1, 0.9, 120, 2, depth)
    ctx.film_clear()
    ctx.render(p)
    want = ctx.film()[0]
    ctx.film_clear()
    b = Batch(0)
    b.add(ctx, p)
    b.tune(1 << 20, streams)
    b.run()
    assert np.array_equal(ctx.film()[0], want)
    b.run()  # the graphs are replayed
    assert np.array_equal(ctx.film()[1], np.full((120, 120), 4, np.float32))
    b.close()


# four waves of 2^18 and 2^20 paths: four and six levels before the loop
@pytest.mark.parametrize("side,depth", [(512, 3), (512, 4), (512, 5), (512, 16), (1024, 5), (1024, 6), (1024, 7), (1024, 16)])
@pytest.mark.parametrize("streams", [0, 1])
def test_repeated_waves(tmp_path, side, depth, streams):
    [(ctx, p)] = _jobs(tmp_path, 1, 0.9, side, 4, depth)
    ctx.film_clear()
    ctx.render(p)
    want = ctx.film()[0]
    ctx.film_clear()
    b = Batch(0)
    b.add(ctx, p)
    b.tune(side * side, streams)
    b.run()
    assert np.array_equal(ctx.film()[0], want)
    b.close()


def _best(f, n=7):
    f()
    times = []
    for _ in range(n):
        t = time.perf_counter()
        f()
        times.append(time.perf_counter() - t)
    return min(times)


# In a bright room most paths live on; rendered together the jobs overlap, so a batch takes less time than its jobs one by one.
@pytest.mark.parametrize("streams", [0, 8])
def test_bright_room_batch_is_not_slower(tmp_path, streams):
    jobs = _jobs(tmp_path, 8, 0.95, 128, 16, 16)

    def one_by_one():
        for ctx, p in jobs:
            ctx.render(p)

    single = _best(one_by_one)
    b = Batch(0)
    for ctx, p in jobs:
        b.add(ctx, p)
    b.tune(1 << 20, streams)
    assert _best(b.run) <= 1.1 * single
    b.close()
