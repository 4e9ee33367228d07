"""Four-wide traversal with quantised planes in scenes and along rays of extreme scale, against the binary SAH
traversal: the same bits of every closest hit's distance, the same any-hit answers.

The scene is a soup of small triangles in the unit cube (over a thousand nodes) and one triangle far away, so
that the nodes near the root span the distance and the others do not."""
import os

import numpy as np
import pytest

from crystal2_gb300 import Context, scenes
from crystal2_gb300 import _native as N

pytestmark = pytest.mark.gpu

TRIS = 4096


def _soup(d, far, spp=1, size=64, others=None):
    tris = scenes.tri_soup_arrays(TRIS, 3).astype(np.float64)
    tris = tris + (tris - tris.mean(axis=1, keepdims=True)) * 4  # edges of some 0.03
    if far:
        tris = np.concatenate([tris, (np.float64([[0, 0, 0], [1, 0, 0], [0, 1, 0]]) * 0.1 + 1.0)[None] * far])
    if others is not None:
        tris = np.concatenate([tris, others])
    tris = tris.astype(np.float32)
    n = np.cross((tris[:, 1] - tris[:, 0]).astype(np.float64), (tris[:, 2] - tris[:, 0]).astype(np.float64))
    n /= np.linalg.norm(n, axis=1, keepdims=True)
    path = os.path.join(d, "soup.obj")
    scenes.write_obj(path, tris.reshape(-1, 3), n.astype(np.float32), np.arange(3 * len(tris)).reshape(-1, 3),
                     np.repeat(np.arange(len(tris))[:, None], 3, axis=1))
    cfg = scenes.config_json(size, size, spp, 4)
    return scenes.write_scene(d, cfg, scenes.camera((0.5, 0.5, -1.5), (0.5, 0.5, 0.5), 45), [scenes.mesh(path, scenes.diffuse((0.5, 0.5, 0.5)))], "soup"), tris


def _axis_rays(tris, seed, zero):
    """Axis-parallel rays at the soup's triangles; the other components are `zero`."""
    rng = np.random.default_rng(seed)
    c = tris[:TRIS].mean(axis=1)
    k = rng.integers(0, 3, TRIS)
    s = rng.choice([-1.0, 1.0], TRIS)
    d = np.full((TRIS, 3), zero, np.float32)
    d[np.arange(TRIS), k] = s
    o = c.copy()
    o[np.arange(TRIS), k] -= np.float32(1.5) * s.astype(np.float32)
    return o.astype(np.float32), d


def _free_rays(seed, n=4096):
    rng = np.random.default_rng(seed)
    d = rng.normal(size=(n, 3))
    return rng.random((n, 3)).astype(np.float32), (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)


def _compare(ctx, o, d, tmax):
    got = {}
    for width in (2, 4):
        ctx.set_traversal(width)
        got[width] = ctx.trace_rays(o, d) + (ctx.trace_rays(o, d, any_hit=True, tmax=tmax),)
    (obj2, t2, any2), (obj4, t4, any4) = got[2], got[4]
    assert np.array_equal(t2.view(np.uint32), t4.view(np.uint32))
    assert np.array_equal(any2, any4)
    return obj2, any2


# scale * 2^100 is infinite from 4.0e8 units on, the offset from 8e8
@pytest.mark.parametrize("far", [0, 1e2, 1e6, 3e8, 4.1e8, 7e8, 9e8, 1e10, 1e18])
def test_axis_parallel_rays_with_a_far_triangle(tmp_path, far):
    (cp, sp), tris = _soup(str(tmp_path), far)
    with Context(0) as ctx:
        ctx.load(cp, sp, tree=N.TREE_SAH)
        for zero in (0.0, -0.0):
            o, d = _axis_rays(tris, 5, zero)
            obj, occluded = _compare(ctx, o, d, np.full(len(o), 1.5, np.float32))
            assert np.mean(obj >= 0) > 0.9 and np.mean(occluded) > 0.3
        o, d = _free_rays(7)
        obj, _ = _compare(ctx, o, d, np.full(len(o), 0.5, np.float32))
        assert np.mean(obj >= 0) > 0.2


# a hit's distance is 1.5 / |d|, up to 2^125 here, against a slab distance of 2^100 or more along the other axes
@pytest.mark.parametrize("far", [0, 1e6])
@pytest.mark.parametrize("length", [-125, -115, -105, -98, -96, -90, -60, 40, 100])
def test_directions_of_any_length(tmp_path, length, far):
    (cp, sp), tris = _soup(str(tmp_path), far)
    with Context(0) as ctx:
        ctx.load(cp, sp, tree=N.TREE_SAH)
        for (o, d), hit in ((_axis_rays(tris, 5, 0.0), 0.5), (_free_rays(7), 0.1)):
            obj, _ = _compare(ctx, o, np.ldexp(d, length), np.ldexp(np.full(len(o), 1.5, np.float32), -length))
            assert length < -100 or np.mean(obj >= 0) > hit  # below, the primitives' own determinants are denormal
        # one component far shorter than the others
        o, d = _free_rays(8)
        d[np.arange(len(d)), np.arange(len(d)) % 3] *= np.float32(2.0 ** -length if length > 0 else 2.0 ** length)
        _compare(ctx, o, d, np.full(len(o), 0.5, np.float32))


# The boxes below the root are as tight as without the far triangle.  The children of the root (and of the few
# nodes that still span the distance) may all be entered, and the tree's levels pair up differently: four nodes
# and a quarter more.
@pytest.mark.parametrize("far", [1e2, 1e4, 1e5, 1e6, 1e9, 1e18])
def test_a_far_triangle_costs_no_culling(tmp_path, far):
    per_ray = []
    for k, dist in enumerate((0, far)):
        d = tmp_path / str(k)
        d.mkdir()
        (cp, sp), _ = _soup(str(d), dist)
        with Context(0) as ctx:
            ctx.load(cp, sp, tree=N.TREE_SAH)
            ctx.set_counting(N.COUNT_TRAVERSAL)
            ctx.render(ctx.render_params())
            s = ctx.stats()
            assert s.rays[N.K_EXTEND] > 4096
            per_ray.append((s.nodes[N.K_EXTEND] / s.rays[N.K_EXTEND], s.prims[N.K_EXTEND] / s.rays[N.K_EXTEND]))
    (nodes0, prims0), (nodes1, prims1) = per_ray
    assert nodes1 <= 1.25 * nodes0 + 4
    assert prims1 <= 1.25 * prims0 + 1


# The soup as a detail among many more, far larger triangles: no more of them are tested than through the binary
# nodes' exact boxes, up to the 8-bit planes' looseness (a tenth without far objects; taken as a quarter and one).
def test_a_detail_among_large_objects(tmp_path):
    rng = np.random.default_rng(4)
    c = rng.uniform(-1e5, 1e5, (40 * TRIS, 1, 3))
    c = c[np.linalg.norm(c[:, 0], axis=1) > 2e4]
    assert len(c) > 32 * TRIS
    (cp, sp), _ = _soup(str(tmp_path), 0, others=c + rng.uniform(-300, 300, (len(c), 3, 3)))
    prims = []
    with Context(0) as ctx:
        ctx.load(cp, sp, tree=N.TREE_SAH)
        ctx.set_counting(N.COUNT_TRAVERSAL)
        for width in (2, 4):
            ctx.set_traversal(width)
            ctx.render(ctx.render_params())
            s = ctx.stats()
            prims.append(s.prims[N.K_EXTEND] / s.rays[N.K_EXTEND])
    assert prims[1] <= 1.25 * prims[0] + 1
