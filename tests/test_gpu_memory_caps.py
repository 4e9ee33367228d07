"""Calls fit the memory caps that they have been known to fit: the least bytes (152 SMs) that each needed when the
context's memory held 16-bit digit tables and a gradient's batch was packed on the host."""
import numpy as np
import pytest

from crystal2_gb300 import Context, scenes
from crystal2_gb300 import _native as N

pytestmark = pytest.mark.gpu

SCENES = {
    "cornell": lambda d: scenes.cornell(d, width=16, height=16, spp=1),
    "material_box": lambda d: scenes.material_box(d, width=24, height=16, spp=1),
    "soup": lambda d: scenes.tri_soup(d, n_tris=300, seed=4),
    "soup2k": lambda d: scenes.tri_soup(d, n_tris=2000, seed=4),
}


def _render(ctx, integrator=N.INTEGRATOR_PATH):
    p = ctx.render_params()
    p.wave_paths = 1
    p.integrator = integrator
    ctx.render(p)


def _samples(n, k):
    return np.random.default_rng(n).normal(size=(n, k)).astype(np.float32)


def _guide(ctx):
    ctx.guide_reset((-1, -1, -1), (1, 1, 1), seed=1)
    return ctx


CALLS = {
    "load": lambda c: None,
    "render": _render,
    "guided": lambda c: _render(c, N.INTEGRATOR_GUIDED),
    "gradient": lambda c: _guide(c).guide_gradient(_samples(100000, 14)),
    "eval": lambda c: _guide(c).guide_eval(_samples(5001, 9)),
    "closest": lambda c: c.trace_rays(_samples(10007, 3), _samples(10007, 3)),
    "any": lambda c: c.trace_rays(_samples(10007, 3), _samples(10007, 3), any_hit=True),
    "halton": lambda c: c.halton(16, 16, *[np.zeros(1001, np.int32)] * 3, 7),
}


@pytest.mark.parametrize("scene,call,cap", [
    ("cornell", "load", 67584), ("cornell", "render", 171520), ("cornell", "guided", 21044480), ("cornell", "gradient", 27041792),
    ("cornell", "eval", 21646336), ("cornell", "closest", 508160), ("cornell", "any", 467968), ("cornell", "halton", 107776),
    ("material_box", "load", 76544), ("material_box", "render", 310528), ("soup", "load", 326144), ("soup", "render", 1702912),
    ("soup2k", "load", 761088), ("soup2k", "render", 2137856),
])
def test_fits(tmp_path, scene, call, cap):
    files = SCENES[scene](str(tmp_path))
    with Context(0, mem_limit_bytes=cap) as ctx:
        ctx.load(*files, tree=N.TREE_SAH)
        CALLS[call](ctx)


# The packed and the raw samples need 120 bytes a sample, the batch alone 64.  The gradient's sums have one order; the
# loss is a sum of atomics, whose last bits differ from call to call, so only its samples' gradient is compared.
@pytest.mark.parametrize("n", [1, 129, 50000])
def test_gradient_of_either_packing(tmp_path, n):
    files = SCENES["cornell"](str(tmp_path))
    s = _samples(n, 14)
    s[:, 3:12] /= np.linalg.norm(s[:, 3:12].reshape(n, 3, 3), axis=2).repeat(3, axis=1)
    s[:, 12:] = np.abs(s[:, 12:]) + 0.1
    got = []
    for cap in (0, 20_000_000 + 100 * n + (1 << 20)):
        with Context(0, mem_limit_bytes=cap) as ctx:
            ctx.load(*files, tree=N.TREE_SAH)
            got.append(_guide(ctx).guide_gradient(s)[0])
    assert np.array_equal(*got)
