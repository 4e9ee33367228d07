"""The explicit gradient is a sum over samples, whatever the number of tiles and warpgroups that share it.

A sample's contribution is the same BF16 product wherever its tile lands; only FP32 sums differ in order.  The
gradient of a batch against the sum of its halves' gradients: each value is a sum of at most n products, so the
difference is within n * 2^-24 of the sum of magnitudes at worst and about sqrt(n) * 2^-24 of it in the 2-norm;
n <= 78000 gives 1.7e-5, taken as 1e-4 of the gradient's norm for the cancellation between samples."""
import numpy as np
import pytest

from crystal2_gb300 import Context, scenes
from crystal2_gb300 import _native as N
from oracle import guide_oracle as G

pytestmark = pytest.mark.gpu


# one sample, edges of a 128-row tile, one tile per warpgroup (304 on 152 SMs) and one more, a second round
@pytest.mark.parametrize("n", [2, 127, 128, 129, 5000, 38912, 38913, 78001])
def test_gradient_adds_up(tmp_path, n):
    cp, sp = scenes.cornell(str(tmp_path), width=8, height=8, spp=1)
    with Context(0) as ctx:
        ctx.load(cp, sp, tree=N.TREE_SAH)
        ctx.guide_reset((-1, -1, -1), (1, 1, 1), seed=3)
        ctx.guide_set_params(G.init_params(2).astype(np.float32))
        x, nr, wo, wi, w, pb = G.random_samples(n, seed=n)
        s = np.concatenate([x, nr, wo, wi, w[:, None], pb[:, None]], axis=1).astype(np.float32)
        g, loss = ctx.guide_gradient(s)
        k = n // 2
        (ga, la), (gb, lb) = ctx.guide_gradient(s[:k]), ctx.guide_gradient(s[k:])
        both = ga.astype(np.float64) + gb
        assert np.linalg.norm(g - both) <= 1e-4 * np.linalg.norm(both)
        wa, wb = s[:k, 12].sum(dtype=np.float64), s[k:, 12].sum(dtype=np.float64)
        assert loss == pytest.approx((la * wa + lb * wb) / (wa + wb), rel=1e-4)


# the step counter and the statistics advance with every Adam step, wherever the last block finishes
@pytest.mark.parametrize("steps", [0, 1, 7])
def test_adam_steps_counted(tmp_path, steps):
    cp, sp = scenes.slit_room(str(tmp_path), width=64, height=36, spp=4, depth=6, hf_res=32)
    with Context(0) as ctx:
        ctx.load(cp, sp, tree=N.TREE_SAH)
        ctx.guide_config(1e-3, 0.7, 0, steps)
        ctx.guide_levels(0)
        p = ctx.render_params()
        p.integrator = N.INTEGRATOR_GUIDED
        p.sample_count = 2
        for wave in range(3):
            ctx.render(p)
            loss, records, done = ctx.guide_stats()
            assert done == steps * (wave + 1)
            assert records > 0 and np.isfinite(loss) and (steps == 0 or loss != 0.0)
        assert np.all(np.isfinite(ctx.guide_params()))
