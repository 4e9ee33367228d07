"""Network outputs do not depend on how many inputs a call has, or on where in a tile one stands.

Each row is one lane of a 128-row tile with its own sums, so the values are the same bits; the counts
cut the last tile, the last warpgroup's turn (640 rows a block) and the last turn of the grid."""
import numpy as np
import pytest

from crystal2_gb300 import Context, scenes
from crystal2_gb300 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 127, 128, 129, 512, 513, 639, 640, 641, 5 * 128 * 152 - 1, 5 * 128 * 152 + 1, 200003])
def test_rows_are_independent(tmp_path, n):
    rng = np.random.default_rng(n)
    unit = rng.normal(size=(2, n, 3))
    unit /= np.linalg.norm(unit, axis=2, keepdims=True)
    x = np.concatenate([rng.uniform(-1, 1, (n, 3)), unit[0], unit[1]], axis=1).astype(np.float32)
    cp, sp = scenes.cornell(str(tmp_path), width=16, height=16, spp=1, depth=2)
    with Context(0) as ctx:
        ctx.load(cp, sp, tree=N.TREE_SAH)
        ctx.guide_reset((-1, -1, -1), (1, 1, 1), seed=7)
        got = ctx.guide_eval(x)
        assert np.isfinite(got).all() and got.std() > 0
        for a in (0, max(0, n - 130), n // 2):
            assert np.array_equal(ctx.guide_eval(x[a:a + 100]), got[a:a + 100])
