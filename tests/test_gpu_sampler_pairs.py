"""Halton dimensions evaluated side by side (pairs of the renderer's draws) against the oracle, bit for bit."""
import numpy as np
import pytest

from crystal2_gb300 import Context, scenes
from crystal2_gb300 import _native as N
from oracle import bindings as B

pytestmark = pytest.mark.gpu


# first pair, small and large bases, the pairs around the end of the tables (dimension 100: hashed)
@pytest.mark.parametrize("dim", [0, 2, 3, 9, 40, 96, 97, 98, 99, 100])
@pytest.mark.parametrize("w,h", [(200, 120), (1920, 1080), (16, 16)])
def test_pairs_match_oracle(tmp_path, dim, w, h):
    cp, sp = scenes.cornell(str(tmp_path), width=w, height=h, spp=4)
    with Context(0) as ctx:
        ctx.load(cp, sp, tree=N.TREE_SAH)
        rng = np.random.default_rng(dim)
        n = 3000
        px, py = rng.integers(0, w, n), rng.integers(0, h, n)
        s = rng.integers(0, 60000, n)  # indices up to just below 2^31
        s[:200] = np.arange(200)       # few digits, among them index 0
        px[0] = py[0] = 0
        want = B.oracle_halton(w, h, px, py, s, dim + 2)[:, dim:dim + 2]
        pair = ctx.sampler_values(px, py, s, dim, two_d=True)
        one = ctx.sampler_values(px, py, s, dim, two_d=False)
        assert np.array_equal(np.ascontiguousarray(pair).view(np.uint32), np.ascontiguousarray(want).view(np.uint32))
        assert np.array_equal(one.view(np.uint32), np.ascontiguousarray(want[:, 0]).view(np.uint32))
