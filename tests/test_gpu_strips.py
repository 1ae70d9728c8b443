"""The resolve pass of frames with somewhat more 32-row tiles than resident
blocks, which takes its tiles whole or in strips of eight rows by how many cells
the triangles reached: sparse, dense and empty frames whose heights end inside a
tile and inside a strip, alone and two in a batch, with record-less pixels, and
with the texture-range error. Against the CPU oracle."""
import numpy as np
import pytest

import cases
from draw_gb300 import scenes as S
from helpers import compare, describe, first_mismatch, gpu_render, oracle_render

pytestmark = pytest.mark.gpu


def _field(width, height, n, seed):
    return S.sphere_field(width=width, height=height, n_spheres=n, slices=16, stacks=9, seed=seed, tex=64, box=12.0)


CASES = {
    # name: (scene, record_limit)
    "sparse": (lambda: S.torus_scene(width=1283, height=717, nu=30, nv=12, tex=64, cam_dist=9.0), 0),
    "sparse_odd": (lambda: S.torus_scene(width=1000, height=681, nu=30, nv=12, tex=64, cam_dist=6.0), 0),
    "dense": (lambda: S.torus_scene(width=1280, height=720, nu=30, nv=12, tex=64, cam_dist=2.2), 0),
    "field": (lambda: _field(1201, 705, 60, 4), 0),
    "no_records": (lambda: S.torus_scene(width=1283, height=717, nu=30, nv=12, tex=64, cam_dist=7.0), 100),
}


def _tiles(d):
    w, h = d.canvas_size
    return ((w + 31) // 32) * ((h + 31) // 32)


@pytest.mark.parametrize("name", sorted(CASES))
def test_strips(name, gpu_ctx, oracle_lib):
    import torch

    make, record_limit = CASES[name]
    desc = make()
    slots = 4 * torch.cuda.get_device_properties(0).multi_processor_count
    assert slots <= _tiles(desc) < 2 * slots
    before = gpu_ctx.get_tuning()
    try:
        gpu_ctx.set_tuning(record_limit=record_limit)
        ref, got = oracle_render(desc, frames=2), gpu_render(desc, gpu_ctx, frames=2)
        st = gpu_ctx.last_stats()
    finally:
        gpu_ctx.set_tuning(**before)
    assert ref[2] == 0 and got[2] == 0 and st["tile_rows"] == 32
    p = compare(ref, got, desc.clear_depth)
    assert p.ok and p.n_covered > 0, f"{describe(p)}; {first_mismatch(ref, got)}"
    assert st["covered_pixels"] == p.n_covered


def test_strips_in_a_batch(gpu_ctx, oracle_lib):
    from draw_gb300 import renderer

    descs = [S.torus_scene(width=700, height=500, nu=24, nv=10, tex=64, cam_dist=8.0), _field(650, 603, 20, 8)]
    built = [renderer.build_scene(d, gpu_ctx) for d in descs]
    empty = renderer.Scene(320, 200, gpu_ctx)
    canvas = renderer.Canvas(320, 200, gpu_ctx)
    canvas.init_depth(7.0)
    gpu_ctx.render_batch([b.scene for b in built] + [empty], [b.canvas for b in built] + [canvas])
    for d, b in zip(descs, built):
        ref = oracle_render(d)
        p = compare(ref, (*b.canvas.read(), 0), d.clear_depth)
        assert p.ok, f"{d.name}: {describe(p)}"
    assert np.all(canvas.read()[1] == 7.0)


def test_strips_texture_range(gpu_ctx, oracle_lib):
    d = cases.texture_range_scene()
    d.width, d.height = 1280, 720
    assert oracle_render(d)[2] == gpu_render(d, gpu_ctx)[2] == 3
