"""Small triangles rasterized by stepping their edge values from pixel to pixel:
boxes of every shape up to 64 pixels, where the steps are exact (near the origin
of the pixel grid) and where they are not (products of coordinates beyond 2^23,
canvases away from the origin), and the vertex marks of a large mesh read in
groups. Against the CPU oracle."""
import numpy as np
import pytest

import cases
from draw_gb300 import scenes as S
from helpers import compare, describe, first_mismatch, gpu_render, oracle_render
from test_gpu_lean import _micro

pytestmark = pytest.mark.gpu


def _specks(side, offset=(0, 0), n=24_000):
    """Triangles of 1 to 17 pixels in each direction, all over a square canvas."""
    rng = np.random.Generator(np.random.PCG64(side))
    half = 10.0 * np.tan(np.radians(30.0))
    at = rng.uniform(-1.0, 1.0, (n, 1, 2))
    size = np.exp(rng.uniform(np.log(1.0), np.log(17.0), (n, 1, 2))) * 2.0 / side
    xy = at + rng.uniform(-0.5, 0.5, (n, 3, 2)) * size
    pos = np.concatenate([xy * half, rng.uniform(-1.0, 1.0, (n, 1, 1)).repeat(3, 1)], 2)
    cross = np.cross(pos[:, 1] - pos[:, 0], pos[:, 2] - pos[:, 1])[:, 2]
    pos[cross < 0] = pos[cross < 0][:, [0, 2, 1]]
    obj = cases._obj(pos.reshape(-1, 3), np.arange(3 * n).reshape(-1, 3), [cases._mat(0)])
    d = cases.flat_scene([obj], width=side, height=side, textures=[S.value_noise_checker(32, 32, 5)])
    d.offset = offset
    return d


CASES = {
    "near": (lambda: _specks(500), {}),
    "near_64": (lambda: _specks(500), dict(small_max_px=64)),
    "far": (lambda: _specks(3200), {}),
    "far_64": (lambda: _specks(3200), dict(small_max_px=64)),
    "offset_64": (lambda: _specks(1600, offset=(-350, 420)), dict(small_max_px=64)),
    "mark_groups": (lambda: _micro(disc_px=14.0), dict(queue_blocks_per_sm=1)),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_small_steps(name, gpu_ctx, oracle_lib):
    make, knobs = CASES[name]
    desc = make()
    before = gpu_ctx.get_tuning()
    try:
        gpu_ctx.set_tuning(**knobs)
        ref, got = oracle_render(desc), gpu_render(desc, gpu_ctx)
        st = gpu_ctx.last_stats()
    finally:
        gpu_ctx.set_tuning(**before)
    assert ref[2] == 0 and got[2] == 0
    assert st["small_triangles"] > 1000
    p = compare(ref, got, desc.clear_depth)
    assert p.ok and p.n_covered > 5000, f"{describe(p)}; {first_mismatch(ref, got)}"
