"""A job that fails part-way, one of its launches refused on the host
(dg_ctx_inject_launch_failure; no GPU fault): the call returns the error, and the
frames after it are those of a context that never failed. The jobs hold every
piece of state that kernels leave to later ones to clear: visibility keys, vertex
marks, counters and fragment lists, and the 2D overlay's lists."""
import numpy as np
import pytest

import cases
from draw_gb300 import scenes as S

pytestmark = pytest.mark.gpu

DG_E_OOM = 7
AWAY, HOME = (0.3, 0.4, 7.0), (0.0, 0.0, 10.0)


def _glass(opaque):
    """Forty transparent layers over `opaque` random triangles (more than 131,072: the
    separate passes instead of the one-kernel front)."""
    rng = np.random.Generator(np.random.PCG64(opaque))
    z = np.linspace(-2.0, 2.0, 40)
    rng.shuffle(z)
    pos, tris = cases._quads([(-2.0, -1.5, 2.0, 1.5, float(v)) for v in z])
    layers = cases._obj(pos, tris, [cases._tmat(0.5, 0), cases._tmat(0.25, 0)], mesh_split=[(50, 0), (30, 1)])
    solid = (rng.uniform(-3.0, 3.0, (opaque, 1, 3)) + rng.uniform(-0.2, 0.2, (opaque, 3, 3))).reshape(-1, 3)
    solid[:, 2] -= 6.0  # behind the layers
    return cases.flat_scene([cases._obj(solid, np.arange(3 * opaque).reshape(-1, 3), [cases._mat(0)]), layers],
                            width=96, height=80, textures=[S.value_noise_checker(32, 32, 5)])


def _read(canvas):
    bgra, depth = canvas.read()
    return bgra.copy(), depth.view(np.uint32).copy()


@pytest.mark.parametrize("opaque", [300, 140_000])
def test_frames_after_a_failed_job(opaque):
    from draw_gb300 import renderer

    ctx = renderer.Context(0)
    try:
        b = renderer.build_scene(_glass(opaque), ctx)
        b.scene.camera._op(7, *HOME)
        for _ in range(2):  # brings the painter's order to rest
            b.scene.render(b.canvas)
        want = _read(b.canvas)
        assert int((want[0][..., 3] == 0).sum()) > 500  # blended pixels
        for before in range(1, 9):
            b.scene.camera._op(7, *AWAY)
            ctx.inject_launch_failure(before)
            with pytest.raises(renderer.DrawError) as err:
                b.scene.render(b.canvas)
            assert err.value.status == DG_E_OOM, before
            b.scene.camera._op(7, *HOME)
            for again in range(3):  # both counter sets
                b.scene.render(b.canvas)
                got = _read(b.canvas)
                assert np.array_equal(want[0], got[0]) and np.array_equal(want[1], got[1]), (before, again)
        ctx.synchronize()  # no error word either
    finally:
        ctx.close()


def test_overlay_after_a_failed_batch():
    from draw_gb300 import renderer

    rng = np.random.Generator(np.random.PCG64(5))
    verts = np.zeros((60, 3, 8), np.float32)
    verts[..., 0], verts[..., 1] = rng.integers(0, 100, (60, 3)), rng.integers(0, 70, (60, 3))
    verts[..., 2:4] = rng.uniform(0.0, 0.9, (60, 3, 2))
    verts[..., 4:7], verts[..., 7] = rng.integers(0, 255, (60, 1, 3)), 0.5
    ctx = renderer.Context(0)
    try:
        tex = rng.integers(0, 255, 16 * 16 * 4).astype(np.uint8)
        atlas = renderer.TextureMap(tex, 16, 16, 4, ctx)
        canvas = renderer.Canvas(100, 70, ctx)
        canvas.init_depth(1.0e9)
        canvas.clear()
        canvas.draw_triangles(verts, atlas)
        want = canvas.read()[0].copy()
        ctx.inject_launch_failure(9)
        with pytest.raises(renderer.DrawError) as err:
            canvas.draw_triangles(verts[::-1].copy(), atlas)
        assert err.value.status == DG_E_OOM
        for _ in range(2):
            canvas.clear()
            canvas.draw_triangles(verts, atlas)
            assert np.array_equal(want, canvas.read()[0])
    finally:
        ctx.close()
