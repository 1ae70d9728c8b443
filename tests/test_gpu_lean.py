"""Frames whose small triangles get no triangle record (at least as many triangles
as pixels, a light/halfway table of at least 128 MB): micro spheres of which some
cross the near plane, so that clipped, larger and small triangles mix, alone,
with the extension modes, under several thresholds, and next to an ordinary frame
in one job. Against the CPU oracle."""
import numpy as np
import pytest

from draw_gb300 import scenes as S
from helpers import compare, describe, first_mismatch, gpu_render, oracle_render

pytestmark = pytest.mark.gpu

LIGHTS = np.array([[0.5, 0.8, 0.5], [-0.6, 0.4, -0.2], [0.4, -0.7, -0.3], [-0.5, -0.5, 0.6], [0.1, 0.9, -0.4],
                   [0.7, -0.2, 0.3], [-0.8, 0.1, 0.2], [0.2, 0.3, -0.9]], np.float32)


def _micro(width=420, height=230, modes=False, disc_px=3.6):
    d = S.micro_sphere_field(width=width, height=height, n_tris=620_000, tex=64, disc_px=disc_px)
    d.lights = LIGHTS
    assert d.n_tris >= width * height and d.objects[0].vertices.shape[0] * len(d.lights) * 32 >= 128 << 20
    if modes:
        d.interpolation, d.textures[0].filter = 1, 1
    return d


CASES = {
    "micro": (_micro, {}),
    "modes": (lambda: _micro(modes=True), {}),
    "larger": (lambda: _micro(disc_px=14.0), {}),
    "threshold_3": (_micro, dict(small_max_px=3)),
    "threshold_4096": (lambda: _micro(disc_px=14.0), dict(small_max_px=4096)),
    "few_records": (lambda: _micro(disc_px=14.0), dict(record_limit=500)),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_lean(name, gpu_ctx, oracle_lib):
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
    assert st["clip_rows"] > 0 and st["launches"] == 6
    # boxes of at most three pixels hold no area: such triangles are dropped
    assert (st["small_triangles"] > 0) == (knobs.get("small_max_px") != 3)
    p = compare(ref, got, desc.clear_depth)
    assert p.ok and p.n_covered > 5000, f"{describe(p)}; {first_mismatch(ref, got)}"


def test_lean_next_to_an_ordinary_frame(gpu_ctx, oracle_lib):
    from draw_gb300 import renderer

    descs = [S.torus_scene(width=300, height=200, nu=30, nv=12, tex=64), _micro(), S.torus_scene(width=160, height=120)]
    built = [renderer.build_scene(d, gpu_ctx) for d in descs]
    for _ in range(2):
        gpu_ctx.render_batch([b.scene for b in built], [b.canvas for b in built])
    for d, b in zip(descs, built):
        ref = oracle_render(d)
        p = compare(ref, (*b.canvas.read(), 0), d.clear_depth)
        assert p.ok, f"{d.name}: {describe(p)}; {first_mismatch(ref, (*b.canvas.read(), 0))}"
