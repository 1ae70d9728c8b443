"""Frames most of whose triangles cross the near or the far plane, some both, so
that whole warps go through the out-of-line clip functions and their records and
light rows fill much of what the resolve pass reads: in the one-kernel front, the
setup pass and the transparent setup, several times. Against the CPU oracle."""
import numpy as np
import pytest

import cases
from draw_gb300 import scenes as S
from helpers import compare, describe, first_mismatch, oracle_render

pytestmark = pytest.mark.gpu


def _shells(n, glass=0, spread=0.12):
    """n opaque and `glass` transparent triangles of random size and direction, half of
    them about the near and half about the far plane, and one in sixteen through both."""
    rng = np.random.Generator(np.random.PCG64(n + glass))

    def mesh(count):
        at = rng.uniform(-1.0, 1.0, (count, 1, 3)) * np.array([0.4, 0.3, 0.08]) + np.array([0.0, 0.0, -0.5])
        far = rng.random(count) < 0.5
        at[far] = at[far] * np.array([4.0, 4.0, 1.0]) + np.array([0.0, 0.0, -0.5])
        pos = at + rng.uniform(-spread, spread, (count, 3, 3))
        both = rng.random(count) < 1.0 / 16.0
        pos[both, 0, 2], pos[both, 1, 2] = -0.3, -1.4
        return pos.reshape(-1, 3).astype(np.float32), np.arange(3 * count, dtype=np.uint32).reshape(-1, 3)

    objects = [cases._obj(*mesh(n), [cases._mat(0)])]
    if glass:
        objects.append(cases._obj(*mesh(glass), [cases._tmat(0.5, 0), cases._tmat(0.25, 0)],
                                  mesh_split=[(glass // 3, 0), (glass - glass // 3, 1)]))
    return S.SceneDesc(120, 90, cam_pos=(0.0, 0.0, 0.0), cam_dir=(0.0, 0.0, -1.0), near=-0.5, far=-1.0, fov_x=60.0,
                       lights=np.array([[2.0, 4.0, 3.0], [-3.0, 1.0, 2.0], [0.5, -2.0, 4.0]], np.float32),
                       textures=[S.value_noise_checker(64, 64, 5)], objects=objects)


CASES = {
    # name: (scene, least rows of opaque clip vertices)
    "front": (lambda: _shells(20_000), 2000),
    "setup": (lambda: _shells(150_000, spread=0.05), 10_000),
    "glass": (lambda: _shells(200, glass=600), 10),
    "glass_behind_setup": (lambda: _shells(140_000, glass=600, spread=0.03), 5000),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_heavy_clipping(name, gpu_ctx, oracle_lib):
    from draw_gb300 import renderer

    make, least = CASES[name]
    desc = make()
    ref = oracle_render(desc)
    assert ref[2] == 0
    for k in range(3):
        b = renderer.build_scene(desc, gpu_ctx)
        b.scene.render(b.canvas)
        got = (*b.canvas.read(), 0)
        assert gpu_ctx.last_stats()["clip_rows"] >= least
        p = compare(ref, got, desc.clear_depth)
        assert p.ok and p.n_covered > 1000, f"render {k}: {describe(p)}; {first_mismatch(ref, got)}"
