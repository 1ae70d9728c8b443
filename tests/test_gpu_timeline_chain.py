"""The DRAW_TIMELINE build shows the kernels that the normal build runs: a small
frame by its one-kernel front, whose vertex and cull passes are points at its
start, and a frame of micro triangles with the setup of its small triangles inside
the setup pass. In a child process, which loads that build (DRAW_GB300_LIB)."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import json, sys
sys.path.insert(0, sys.argv[1]); sys.path.insert(0, sys.argv[1] + "/tests")
from draw_gb300 import renderer, scenes as S
from test_gpu_lean import _micro
ctx = renderer.Context(0)
out = {}
for name, d in [("torus", S.torus_scene()), ("micro", _micro())]:
    b = renderer.build_scene(d, ctx)
    for _ in range(3):
        b.scene.render(b.canvas)
    ctx.timeline()
    b.scene.render(b.canvas)
    out[name] = dict(timeline=ctx.timeline(), launches=ctx.last_stats()["launches"])
ctx.close()
print(json.dumps(out))
"""


def test_timeline_of_the_front_and_of_micro_triangles():
    from draw_gb300 import _build

    lib = _build.build(timeline=True)
    env = dict(os.environ, DRAW_GB300_LIB=lib)
    r = subprocess.run([sys.executable, "-c", CHILD, ROOT], capture_output=True, text=True, env=env, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    res = json.loads(r.stdout.strip().splitlines()[-1])
    torus, micro = res["torus"], res["micro"]
    assert torus["launches"] == 3 and micro["launches"] == 6
    t = torus["timeline"]
    assert t["vertex"][0] == t["vertex"][3] == t["cull"][0] == t["cull"][3]
    assert t["setup_raster"][3] > t["setup_raster"][0] and t["queue_raster"][1] >= t["setup_raster"][3]
    # 284,000 list entries are most of this frame's setup: they begin right after the cull
    t = micro["timeline"]
    cull_end, (_, first_wait, _, end) = t["cull"][3], t["setup_raster"]
    assert cull_end <= first_wait and first_wait - cull_end < 0.25 * (end - cull_end), t
