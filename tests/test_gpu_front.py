"""The one-kernel front of small jobs (vertex, cull and setup of at most 131,072
triangles) against the three separate passes, which the same scene takes as part
of a captured batch: frames bit-identical, and equal to the CPU oracle, and the
statistics of a batch of two the sum of theirs. At the sizes where the front's
blocks and its limit end, on clipped geometry, and with several objects per frame;
and the descriptors that travel with the first kernel at the numbers of frames and
objects where their room ends."""
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
    assert stats["launches"] == (3 if desc.n_tris <= 131072 else 5)
    assert both["launches"] == (3 if desc.n_tris + cases.tie_rule_scene().n_tris <= 131072 else 5)
    for k in keys[:-1]:
        assert stats[k] + other[k] == both[k], (k, stats[k], other[k], both[k])
    graph = gpu_ctx.batch([a.scene, b.scene], [a.canvas, b.canvas])  # the separate passes
    try:
        graph.render()
        replayed = a.canvas.read()
    finally:
        graph.close()
    assert np.array_equal(alone[0], replayed[0])
    assert np.array_equal(alone[1].view(np.uint32), replayed[1].view(np.uint32))


def _several(objects, n):
    """A frame of several objects, another one for each n."""
    parts = []
    for k in range(objects):
        c, s = np.cos(0.7 * k + n), np.sin(1.1 * k + n)
        z = -0.3 * k
        parts.append(cases._obj([[c - 2, s - 2, z], [c + 2, s - 2, z], [c, s + 2, z + 0.5 * c]], [[0, 1, 2]],
                                [cases._mat(0)]))
    return cases.flat_scene(parts, width=48 + n % 5, height=40 + n % 3)


# frames, objects per frame: one frame of up to 4 objects, 16 frames with 24 objects in all, 48 with 72, more
@pytest.mark.parametrize("frames,objects,tris", [(1, 4, 1), (1, 5, 1), (1, 24, 1), (1, 25, 1), (1, 72, 1), (1, 73, 1),
                                                 (2, 12, 1), (2, 13, 1), (16, 1, 1), (17, 1, 1), (48, 1, 1), (49, 1, 1),
                                                 (3, 1, 70_000), (13, 1, 10_000)])
def test_descriptors_with_the_first_kernel(frames, objects, tris, gpu_ctx, oracle_lib):
    from draw_gb300 import renderer

    descs = [_several(objects, n) if tris == 1 else _triangles(tris + n) for n in range(frames)]
    built = [renderer.build_scene(d, gpu_ctx) for d in descs]
    for _ in range(2):
        gpu_ctx.render_batch([b.scene for b in built], [b.canvas for b in built])
    small = frames <= 48 and frames * objects <= 72 and sum(d.n_tris for d in descs) <= 131072
    assert gpu_ctx.last_stats()["launches"] == (3 if small else 5)
    for d, b in zip(descs, built):
        ref, got = oracle_render(d), (*b.canvas.read(), 0)
        p = compare(ref, got, d.clear_depth)
        assert p.ok, f"{d.name}: {describe(p)}; {first_mismatch(ref, got)}"
