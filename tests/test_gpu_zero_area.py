"""Triangles without area on the pixel grid (collinear, coincident, one-pixel) are
dropped before the setup where that is proved to cover nothing: dense meshes in
small frames, with the canvas away from the origin of the pixel grid and with
coordinates too large for the proof, equal the CPU oracle's frames, as single
frames and in a batch; most of the dense mesh is dropped."""
import numpy as np
import pytest

import cases
from draw_gb300 import scenes as S
from helpers import compare, describe, first_mismatch, gpu_render, oracle_render

pytestmark = pytest.mark.gpu


def _dense(width, height, tris, offset=(0, 0), scale=1.0):
    pos, nrm, uv, tri = S.mesh_for_tris("sphere", tris)
    obj = S.ObjectDesc((pos * scale).astype(np.float32), nrm, uv, [S.MeshDesc(S._tris9(tri), 0)], [cases._mat(0)])
    return S.SceneDesc(width, height, cam_pos=(0.3, 0.9, 2.9), cam_dir=(-0.3, -0.9, -2.9), near=-0.5, far=-100.0,
                       fov_x=60.0, lights=np.array([[2.0, 4.0, 3.0]], np.float32), offset=offset,
                       textures=[S.value_noise_checker(64, 64, 5)], objects=[obj])


def _points(reach):
    """Triangles whose corners lie on one pixel row, column or diagonal, or on one
    pixel, next to ordinary ones; `reach` spreads them beyond the canvas."""
    rng = np.random.Generator(np.random.PCG64(int(reach)))
    half = 10.0 * np.tan(np.radians(30.0))
    n = 300
    a = rng.uniform(-reach, reach, (n, 2))
    d = rng.uniform(-1.0, 1.0, (n, 2)) * reach
    d[::4, 0] = 0.0
    d[1::4, 1] = 0.0
    d[2::4, 1] = d[2::4, 0]
    xy = np.stack([a, a + d, a + d * rng.uniform(-1.0, 1.0, (n, 1))], 1)
    xy[3::4] = a[3::4, None] + rng.uniform(-0.004, 0.004, (len(a[3::4]), 3, 2))
    xy[::9] = a[::9, None] + rng.uniform(-0.3, 0.3, (len(a[::9]), 3, 2))
    pos = np.concatenate([xy * half, rng.uniform(-1.0, 1.0, (n, 1, 1)).repeat(3, 1)], 2)
    cross = np.cross(pos[:, 1] - pos[:, 0], pos[:, 2] - pos[:, 1])[:, 2]
    pos[cross < 0] = pos[cross < 0][:, [0, 2, 1]]
    obj = cases._obj(pos.reshape(-1, 3), np.arange(3 * n).reshape(-1, 3), [cases._mat(0)])
    return cases.flat_scene([obj], width=160, height=160, textures=[S.value_noise_checker(32, 32, 5)])


CASES = {
    "dense": lambda: _dense(150, 120, 60_000),
    "dense_large_job": lambda: _dense(150, 120, 200_000),
    "offset": lambda: _dense(150, 120, 20_000, offset=(37, -21)),
    "points_near": lambda: _points(1.2),
    "points_far": lambda: _points(400.0),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_zero_area(name, gpu_ctx, oracle_lib):
    from draw_gb300 import renderer

    desc = CASES[name]()
    ref, got = oracle_render(desc), gpu_render(desc, gpu_ctx)
    st = gpu_ctx.last_stats()
    assert ref[2] == 0 and got[2] == 0
    p = compare(ref, got, desc.clear_depth)
    assert p.ok, f"{describe(p)}; {first_mismatch(ref, got)}"
    assert p.n_covered > 0 or name == "points_far"  # none of the far ones reaches a pixel
    if name.startswith("dense"):
        assert st["survivors"] < 0.35 * desc.n_tris  # about half of them face the camera
    a, b = renderer.build_scene(desc, gpu_ctx), renderer.build_scene(cases.tie_rule_scene(), gpu_ctx)
    gpu_ctx.render_batch([a.scene, b.scene], [a.canvas, b.canvas])  # the separate passes
    q = compare(ref, (*a.canvas.read(), 0), desc.clear_depth)
    assert q.ok, describe(q)
