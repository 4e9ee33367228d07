"""Four-wide traversal (quantised and exact planes, ray replacement) against the binary SAH traversal.

Both run the same exact primitive tests, so a closest hit's distance has the same bits and an any-hit
answer is the same; only the object may differ, where two objects are hit at one distance."""
import numpy as np
import pytest

from crystal2_gb300 import Context, scenes
from crystal2_gb300 import _native as N

pytestmark = pytest.mark.gpu


def _rays(n, lo, hi, seed):
    """Random rays through the box, a third of them axis-parallel (zero direction components), some from far away."""
    rng = np.random.default_rng(seed)
    lo, hi = np.asarray(lo, np.float64), np.asarray(hi, np.float64)
    o = lo + (hi - lo) * rng.random((n, 3))
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    k = np.arange(n)
    par = k % 3 == 0
    d[par] = np.eye(3)[rng.integers(0, 3, par.sum())] * rng.choice([-1.0, 1.0], (par.sum(), 1))
    far = k % 7 == 0
    o[far] -= d[far] * 50.0 * np.max(hi - lo)
    plane = k % 5 == 0  # one zero component
    d[plane, rng.integers(0, 3, plane.sum())] = 0.0
    d[np.all(d == 0, axis=1)] = (0.0, 1.0, 0.0)
    return o.astype(np.float32), d.astype(np.float32), (rng.random(n) * 2 * np.max(hi - lo)).astype(np.float32)


def _compare(ctx, n, lo, hi, seed):
    o, d, tmax = _rays(n, lo, hi, seed)
    got = {}
    for width in (2, 4):
        ctx.set_traversal(width)
        got[width] = ctx.trace_rays(o, d) + (ctx.trace_rays(o, d, any_hit=True, tmax=tmax),)
    obj2, t2, any2 = got[2]
    obj4, t4, any4 = got[4]
    assert np.array_equal(t2.view(np.uint32), t4.view(np.uint32))
    assert np.mean(obj2 != obj4) <= 0.01  # equal distances only (the distances above are the same)
    assert np.array_equal(any2, any4)
    return obj2


# the number of primitives crosses the limit of the exact-plane nodes; one triangle is a single leaf
@pytest.mark.parametrize("tris", [1, 2, 3, 24, 40, 64, 1000])
def test_soup_sizes(tmp_path, tris):
    cp, sp = scenes.tri_soup(str(tmp_path), n_tris=tris, seed=tris)
    with Context(0) as ctx:
        ctx.load(cp, sp, tree=N.TREE_SAH)
        _compare(ctx, 20000, (0, 0, 0), (1, 1, 1), tris)


# fewer rays than threads are spread over the warps; more are refilled
@pytest.mark.parametrize("n", [1, 31, 33, 1000, 40000, 155647, 155649, 400001])
def test_ray_counts(tmp_path, n):
    cp, sp = scenes.tri_soup(str(tmp_path), n_tris=2000, seed=9)
    with Context(0) as ctx:
        ctx.load(cp, sp, tree=N.TREE_SAH)
        _compare(ctx, n, (0, 0, 0), (1, 1, 1), n)


# flat axis-aligned walls, spheres and disks, under both accelerators' shadow semantics
@pytest.mark.parametrize("accel", ["BVH", "Brute"])
@pytest.mark.parametrize("scene", ["material_box", "slit_room"])
def test_walls_and_quadrics(tmp_path, scene, accel):
    if scene == "material_box":
        cp, sp = scenes.material_box(str(tmp_path), accel=accel)
        box = ((-2, 0, -2), (2, 3, 2))
    else:
        cp, sp = scenes.slit_room(str(tmp_path), width=64, height=36, hf_res=48, accel=accel)
        box = ((-5, 0, -5), (5, 4, 6))
    with Context(0) as ctx:
        ctx.load(cp, sp, tree=N.TREE_SAH)
        hits = _compare(ctx, 60000, *box, 3)
        assert np.mean(hits >= 0) > 0.3
