"""First calls of several threads at once, in a new process: launch sizes are found once and no thread sees half of them."""
import os
import subprocess
import sys

import pytest

from crystal2_gb300 import scenes

pytestmark = pytest.mark.gpu

WORK = """
import sys, threading
import numpy as np
from crystal2_gb300 import Context
from crystal2_gb300 import _native as N
kind, cp, sp = sys.argv[1:4]
rng = np.random.default_rng(1)
o, d = rng.random((500, 3)), rng.normal(size=(500, 3))
ctxs = [Context(0) for _ in range(8)]
for c in ctxs:
    c.load(cp, sp, tree=N.TREE_SAH)
    if kind == "guide":
        c.guide_reset((-1, -1, -1), (1, 1, 1), seed=1)
gate, got = threading.Barrier(8), [None] * 8

def call(k):
    c = ctxs[k]
    gate.wait()
    try:
        if kind == "rays":
            got[k] = c.trace_rays(o, d, any_hit=True) if k % 2 else c.trace_rays(o, d)[0]
        elif kind == "guide":
            got[k] = c.guide_eval(np.concatenate([o, d, d], axis=1))
        else:
            c.render(c.render_params())
            got[k] = c.film()[0]
    except Exception as e:
        got[k] = repr(e)

threads = [threading.Thread(target=call, args=(k,)) for k in range(8)]
[t.start() for t in threads]
[t.join() for t in threads]
for k in range(8):
    assert isinstance(got[k], np.ndarray), got[k]
    assert np.array_equal(got[k], got[k % 2 if kind == "rays" else 0])
assert np.any(got[0]) and np.any(got[1])
"""


@pytest.mark.parametrize("kind", ["rays", "render", "guide"])
def test_threads_first_calls(tmp_path, kind):
    cp, sp = scenes.tri_soup(str(tmp_path), n_tris=2000, seed=4) if kind == "rays" else scenes.cornell(str(tmp_path), width=120, height=90, spp=2)
    for _ in range(6):
        r = subprocess.run([sys.executable, "-c", WORK, kind, cp, sp], capture_output=True, text=True, timeout=120,
                           cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
        assert r.returncode == 0, r.stderr[-2000:]
