"""Renders that the caller captures on its own stream (dg_ctx_set_stream) and
replays: every replay starts a job of its own, whatever ran before it, so its
frame and its counters are those of a plain render, and plain renders after it
are not disturbed. At sizes that take the one-kernel front, the separate passes,
a batch, strips in the resolve pass, and a transparent pass."""
import numpy as np
import pytest

import cases
from draw_gb300 import scenes as S

pytestmark = pytest.mark.gpu


def _sphere(n, w=320, h=200):
    pos, nrm, uv, tri = S.mesh_for_tris("sphere", n)
    obj = S.ObjectDesc(pos, nrm, uv, [S.MeshDesc(S._tris9(tri), 0)], [cases._mat(0)])
    return S.SceneDesc(w, h, cam_pos=(0.4, 1.0, 2.6), cam_dir=(-0.4, -1.0, -2.6), near=-0.5, far=-100.0, fov_x=60.0,
                       lights=np.array([[2.0, 4.0, 3.0]], np.float32), textures=[S.value_noise_checker(64, 64, 5)],
                       objects=[obj])


def _glass():
    pos, tris = cases._quads([(-2.0, -2.0, 2.0, 2.0, 1.0), (-3.0, -1.0, 1.0, 2.0, 2.0)])
    glass = cases._obj(pos, tris, [cases._tmat(0.5, 0)])
    bp, bt = cases._quads([(-1.0, -1.0, 2.0, 1.5, 0.1)])
    return cases.flat_scene([cases._obj(bp, bt, [cases._mat(0)]), glass], width=96, height=80,
                            textures=[S.value_noise_checker(32, 32, 5)])


CASES = {
    "front": lambda: [_sphere(3000)],
    "passes": lambda: [_sphere(200_000)],
    "batch": lambda: [_sphere(3000), _sphere(90_000), _sphere(60_000, 200, 160)],
    "strips": lambda: [S.torus_scene(width=1280, height=720, nu=30, nv=12, tex=64, cam_dist=6.0)],
    "glass": lambda: [_glass()],
}
KEYS = ["survivors", "triangle_records", "queued_triangles", "small_triangles", "covered_pixels", "clip_rows"]


def _read(built):
    out = []
    for b in built:
        bgra, depth = b.canvas.read()
        out.append((bgra.copy(), depth.view(np.uint32).copy()))
    return out


def _equal(a, b):
    return all(np.array_equal(x[0], y[0]) and np.array_equal(x[1], y[1]) for x, y in zip(a, b))


@pytest.mark.parametrize("name", sorted(CASES))
def test_replays(name, oracle_lib):
    import torch
    from draw_gb300 import renderer

    ctx = renderer.Context(0)
    try:
        stream = torch.cuda.Stream()
        ctx.set_stream(stream.cuda_stream)
        built = [renderer.build_scene(d, ctx) for d in CASES[name]()]

        def render():
            ctx.render_batch([b.scene for b in built], [b.canvas for b in built])

        for _ in range(2):  # allocates the scratch, and brings a painter's order to rest
            render()
        want = _read(built)
        stats = {k: ctx.last_stats()[k] for k in KEYS}
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
            render()
        for _ in range(7):
            for b in built:
                b.canvas.clear()
            with torch.cuda.stream(stream):
                graph.replay()
            assert _equal(want, _read(built))
            got = ctx.last_stats()
            assert {k: got[k] for k in KEYS} == stats
        for _ in range(6):  # every staging buffer and both counter sets
            render()
            assert _equal(want, _read(built))
            got = ctx.last_stats()
            assert {k: got[k] for k in KEYS} == stats
        with torch.cuda.stream(stream):
            graph.replay()
        assert _equal(want, _read(built))
        torch.cuda.synchronize()
        del graph
    finally:
        ctx.set_stream(None)
        ctx.close()


def test_overlay_is_refused_in_a_capture(oracle_lib):
    """A graph would read the call's staging buffer at every replay: refused, and the
    context works on."""
    import torch
    from draw_gb300 import renderer

    ctx = renderer.Context(0)
    try:
        stream = torch.cuda.Stream()
        ctx.set_stream(stream.cuda_stream)
        canvas = renderer.Canvas(64, 48, ctx)
        canvas.init_depth(1.0e9)
        verts = np.zeros((1, 3, 8), np.float32)
        verts[0, :, :2] = [[2, 2], [60, 2], [2, 40]]
        verts[..., 4:7], verts[..., 7] = 200.0, 0.5
        atlas = renderer.TextureMap(np.full(8 * 8 * 4, 255, np.uint8), 8, 8, 4, ctx)
        canvas.draw_triangles(verts, atlas)  # allocates the scratch
        before = canvas.read()[0].copy()
        graph = torch.cuda.CUDAGraph()
        with pytest.raises(renderer.DrawError) as err:
            with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
                torch.zeros(1, device="cuda")  # the graph is not empty
                canvas.draw_triangles(verts, atlas)
        assert err.value.status == 6  # DG_E_CUDA
        assert np.array_equal(before, canvas.read()[0])
        canvas.draw_triangles(verts, atlas)
        assert not np.array_equal(before, canvas.read()[0])
        torch.cuda.synchronize()
    finally:
        ctx.set_stream(None)
        ctx.close()
