"""Strips or whole tiles are decided by the number of reached cells, which the
queue pass counts before it lets the resolve pass start: every block of the
resolve pass must see the complete count. Under queue grids of one wave and less,
a frame just below and one just above the threshold, and a batch of many small
frames, several times into the same canvases. Against the CPU oracle."""
import numpy as np
import pytest

from draw_gb300 import scenes as S
from helpers import compare, describe, first_mismatch, oracle_render

pytestmark = pytest.mark.gpu


def _slots():
    import torch

    return 4 * torch.cuda.get_device_properties(0).multi_processor_count


def _reached(depth, clear):
    """32x32 cells (rows from the bottom, as the depth rows) that hold a fragment."""
    h, w = depth.shape
    pad = np.full(((h + 31) // 32 * 32, (w + 31) // 32 * 32), False)
    pad[:h, :w] = depth != clear
    return int(pad.reshape(pad.shape[0] // 32, 32, -1, 32).any(axis=(1, 3)).sum())


def _torus(cam_dist):
    return S.torus_scene(width=1280, height=720, nu=30, nv=12, tex=64, cam_dist=cam_dist)


@pytest.mark.parametrize("blocks", [1, 4, 12])
@pytest.mark.parametrize("side", ["below", "above"])
def test_threshold_sides(side, blocks, gpu_ctx, oracle_lib):
    from draw_gb300 import renderer

    # the camera distance whose frame is nearest to the threshold on its side
    # (reached cells also count boxes' corners, so the frames bracket it with some room)
    want = _slots() // 2
    frames = []
    for dist in np.arange(2.0, 6.01, 0.25):
        d = _torus(float(dist))
        ref = oracle_render(d)
        frames.append((_reached(np.asarray(ref[1]).reshape(720, 1280), d.clear_depth), d, ref))
    lower = [f for f in frames if f[0] < want * 0.9]
    upper = [f for f in frames if f[0] >= want]
    n, d, ref = max(lower, key=lambda f: f[0]) if side == "below" else min(upper, key=lambda f: f[0])
    assert _slots() <= 40 * 23 < 2 * _slots()
    before = gpu_ctx.get_tuning()
    try:
        gpu_ctx.set_tuning(queue_blocks_per_sm=blocks)
        b = renderer.build_scene(d, gpu_ctx)
        for k in range(12):
            b.scene.render(b.canvas)
            p = compare(ref, (*b.canvas.read(), 0), d.clear_depth)
            assert p.ok and p.n_covered > 0, f"frame {k}, {n} cells: {describe(p)}; {first_mismatch(ref, (*b.canvas.read(), 0))}"
            assert gpu_ctx.last_stats()["covered_pixels"] == p.n_covered
    finally:
        gpu_ctx.set_tuning(**before)


@pytest.mark.parametrize("blocks", [1, 4])
def test_many_frames(blocks, gpu_ctx, oracle_lib):
    from draw_gb300 import renderer

    descs = [S.torus_scene(width=192, height=160, nu=16, nv=8, tex=64, cam_dist=3.0 + 0.2 * i) for i in range(26)]
    assert _slots() <= 26 * 6 * 5 < 2 * _slots()
    refs = [oracle_render(d) for d in descs]
    before = gpu_ctx.get_tuning()
    try:
        gpu_ctx.set_tuning(queue_blocks_per_sm=blocks)
        built = [renderer.build_scene(d, gpu_ctx) for d in descs]
        for k in range(8):
            gpu_ctx.render_batch([b.scene for b in built], [b.canvas for b in built])
            for i, (d, ref, b) in enumerate(zip(descs, refs, built)):
                p = compare(ref, (*b.canvas.read(), 0), d.clear_depth)
                assert p.ok, f"pass {k}, frame {i}: {describe(p)}"
    finally:
        gpu_ctx.set_tuning(**before)
