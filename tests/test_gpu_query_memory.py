"""Queries that share one kept block of device memory answer as in a fresh context.

Sizes below and above the block's limit (16 MB: 419430 rays of 40 bytes), growing and shrinking, of
different kinds in turn, with and without a memory cap (which keeps nothing)."""
import numpy as np
import pytest

from crystal2_gb300 import Context, scenes
from crystal2_gb300 import _native as N

pytestmark = pytest.mark.gpu


def _ask(ctx, kind, n):
    rng = np.random.default_rng([n, len(kind)])
    if kind == "halton":
        px = rng.integers(0, 64, n)
        return (ctx.halton(64, 64, px, px[::-1], rng.integers(0, 99, n), 7),)
    if kind == "camera":
        return ctx.camera_rays(rng.random((n, 2)))
    o = rng.uniform(-1, 1, (n, 3))
    d = rng.normal(size=(n, 3))
    if kind == "any":
        return (ctx.trace_rays(o, d, any_hit=True, tmax=rng.random(n) * 2),)
    return ctx.trace_rays(o, d)


@pytest.mark.parametrize("cap", [0, 256 << 20])
def test_shared_block(tmp_path, cap):
    cp, sp = scenes.tri_soup(str(tmp_path), n_tris=300, seed=4)
    asked = [("closest", 1), ("any", 333), ("halton", 1000), ("closest", 419430), ("any", 419431), ("camera", 70), ("any", 500001),
             ("closest", 33), ("halton", 5)]
    with Context(0, mem_limit_bytes=cap) as shared:
        shared.load(cp, sp, tree=N.TREE_SAH)
        for kind, n in asked:
            got = _ask(shared, kind, n)
            with Context(0) as fresh:
                fresh.load(cp, sp, tree=N.TREE_SAH)
                want = _ask(fresh, kind, n)
            for a, b in zip(got, want):
                assert np.array_equal(a, b)
