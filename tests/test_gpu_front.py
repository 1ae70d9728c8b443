"""The one-kernel front of small jobs (vertex, cull and setup of at most 131,072
triangles of one frame) against the three separate passes, which the same scene
takes as part of a two-frame batch: both frames bit-identical, the statistics
equal, and equal to the CPU oracle. At the sizes where the front's blocks and its
limit end, on clipped geometry, and with several objects per frame."""
import numpy as np
import pytest

import cases
from draw_gb300 import scenes as S
from helpers import compare, describe, first_mismatch, oracle_render

pytestmark = pytest.mark.gpu


def _triangles(n):
    """The first n triangles of a sphere seen from outside."""
    pos, nrm, uv, tri = S.mesh_for_tris("sphere", max(n, 200) + 600)
    assert len(tri) >= n
    rng = np.random.Generator(np.random.PCG64(n))
    t9 = S._tris9(tri[np.sort(rng.permutation(len(tri))[:n])])
    obj = S.ObjectDesc(pos, nrm, uv, [S.MeshDesc(t9, 0)], [cases._mat(0)])
    return S.SceneDesc(200, 160, cam_pos=(0.4, 1.0, 2.6), cam_dir=(-0.4, -1.0, -2.6), near=-0.5, far=-100.0, fov_x=60.0,
                       lights=np.array([[2.0, 4.0, 3.0]], np.float32), textures=[S.value_noise_checker(64, 64, 5)],
                       objects=[obj])


CASES = {
    "tris_1": lambda: _triangles(1),
    "tris_31": lambda: _triangles(31),
    "tris_127": lambda: _triangles(127),
    "tris_129": lambda: _triangles(129),
    "tris_4000": lambda: _triangles(4000),
    "tris_131072": lambda: _triangles(131072),
    "tris_131073": lambda: _triangles(131073),
    "clip": cases.clip_scene,
    "degenerate": cases.degenerate_scene,
    "multi_object": cases.multi_object_scene,
    "crossing_field": lambda: S.sphere_field(width=320, height=200, n_spheres=60, slices=20, stacks=11, tex=64, box=3.0),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_front_equals_separate_passes(name, gpu_ctx, oracle_lib):
    from draw_gb300 import renderer

    desc = CASES[name]()
    a, b = renderer.build_scene(desc, gpu_ctx), renderer.build_scene(cases.tie_rule_scene(), gpu_ctx)
    keys = ["survivors", "triangle_records", "queued_triangles", "queued_units", "small_triangles", "covered_pixels",
            "clip_rows", "launches"]
    a.scene.render(a.canvas)
    alone = (*a.canvas.read(), 0)
    stats = gpu_ctx.last_stats()
    b.scene.render(b.canvas)
    other = gpu_ctx.last_stats()
    gpu_ctx.render_batch([a.scene, b.scene], [a.canvas, b.canvas])
    batched = (*a.canvas.read(), 0)
    both = gpu_ctx.last_stats()
    ref = oracle_render(desc)
    p = compare(ref, alone, desc.clear_depth)
    assert p.ok, f"{describe(p)}; {first_mismatch(ref, alone)}"
    assert np.array_equal(alone[0], batched[0])
    assert np.array_equal(alone[1].view(np.uint32), batched[1].view(np.uint32))
    assert stats["launches"] == (3 if desc.n_tris <= 131072 else 5) and both["launches"] == 5
    for k in keys[:-1]:
        assert stats[k] + other[k] == both[k], (k, stats[k], other[k], both[k])
