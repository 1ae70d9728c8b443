"""The queue pass's row spans against the CPU oracle: seeded triangles from
slivers to boxes far larger than the canvas (whose edge constants leave the
range of the span estimate), drawn into wide, tall, tiny and ordinary canvases
under item sizes from the smallest to the largest, with every triangle sent
through the queue. Depth bit-exact, colour within 1 LSB."""
import numpy as np
import pytest

import cases
from draw_gb300 import scenes as S
from helpers import compare, describe, first_mismatch, gpu_render, oracle_render

pytestmark = pytest.mark.gpu


def _scene(width, height, reach, n=120, seed=0):
    """n triangles facing the camera whose corners spread over `reach` times the frame."""
    rng = np.random.Generator(np.random.PCG64(seed + int(reach * 8) + width))
    half = 10.0 * np.tan(np.radians(30.0))
    size = np.exp(rng.uniform(np.log(0.02), np.log(reach), (n, 1, 1)))
    centre = rng.uniform(-1.0, 1.0, (n, 1, 2)) * min(reach, 1.5)
    xy = (centre + rng.uniform(-1.0, 1.0, (n, 3, 2)) * size) * half * np.array([1.0, height / width])
    xy[::7, 2] = xy[::7, 0] + rng.uniform(-0.01, 0.01, (len(xy[::7]), 2))  # slivers
    xy[3::11, 1, 1] = xy[3::11, 0, 1]  # a horizontal edge
    xy[5::13, 1, 0] = xy[5::13, 0, 0]  # a vertical edge
    pos = np.concatenate([xy, rng.uniform(-1.0, 1.0, (n, 1, 1)).repeat(3, 1)], 2)
    a, b, c = pos[:, 0, :2], pos[:, 1, :2], pos[:, 2, :2]
    away = ((b - a)[:, 0] * (c - b)[:, 1] - (b - a)[:, 1] * (c - b)[:, 0]) < 0
    pos[away] = pos[away][:, [0, 2, 1]]
    obj = cases._obj(pos.reshape(-1, 3), np.arange(3 * n).reshape(-1, 3), [cases._mat(0)],
                     uvs=np.tile(np.array([[0.2, 0.3, 0], [0.8, 0.2, 0], [0.5, 0.9, 0]], np.float32), (n, 1)))
    return cases.flat_scene([obj], width=width, height=height, textures=[S.value_noise_checker(32, 32, 5)])


@pytest.mark.parametrize("item_units", [1, 3, 8, 256])
@pytest.mark.parametrize("reach", [0.2, 2.0, 60.0, 40000.0])
@pytest.mark.parametrize("size", [(500, 300), (2011, 7), (9, 1500), (33, 65)])
def test_row_spans(size, reach, item_units, gpu_ctx, oracle_lib):
    desc = _scene(*size, reach)
    before = gpu_ctx.get_tuning()
    try:
        gpu_ctx.set_tuning(item_units=item_units, small_max_px=0)
        ref, got = oracle_render(desc), gpu_render(desc, gpu_ctx)
        queued = gpu_ctx.last_stats()["queued_triangles"]
    finally:
        gpu_ctx.set_tuning(**before)
    assert ref[2] == 0 and got[2] == 0 and queued > 0
    p = compare(ref, got, desc.clear_depth)
    assert p.ok, f"{describe(p)}; {first_mismatch(ref, got)}"
