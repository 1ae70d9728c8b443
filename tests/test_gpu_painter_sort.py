"""The painter's sort of transparent meshes around the edges of its one-block
form (powers of two, 4,096 triangles, a job with one larger mesh): after each
frame the persistent order of every mesh equals the oracle's."""
import numpy as np
import pytest

import cases
from draw_gb300 import scenes as S
from test_gpu_transparent import _oracle_objects

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(1,), (2, 63), (64, 65), (0, 1023, 1024, 3), (4096,), (5, 4097, 100)])
def test_order_of_mesh_sizes(sizes, gpu_ctx, oracle_lib):
    from draw_gb300 import renderer

    rng = np.random.Generator(np.random.PCG64(sum(sizes)))
    n = sum(sizes)
    base = rng.uniform(-3.0, 3.0, (n, 1, 3))
    base[::3] = base[0]  # groups at exactly equal distances: the previous order decides
    pos = (base + np.array([[0.0, 0.0, 0.0], [0.05, 0.0, 0.0], [0.0, 0.05, 0.0]])).reshape(-1, 3)
    obj = cases._obj(pos, np.arange(3 * n).reshape(-1, 3), [cases._tmat(0.5, 0)], mesh_split=[(s, 0) for s in sizes])
    desc = cases.flat_scene([obj], width=48, height=40, textures=[S.value_noise_checker(32, 32, 5)])
    o, s, c, oids = _oracle_objects(desc)
    b = renderer.build_scene(desc, gpu_ctx)
    for cam in ((0.0, 0.0, 10.0), (1.0, -2.0, 9.0), (0.0, 0.0, 10.0)):
        o.camera_op(s, 7, cam)
        b.scene.camera._op(7, *cam)
        assert o.render(s, c) == 0
        b.scene.render(b.canvas)
        gpu_ctx.synchronize()
        for mi, size in enumerate(sizes):
            want = o.transparent_tris(oids[0], mi, size)
            assert np.array_equal(want, b.objects[0].transparent_triangles(mi)), (sizes, mi, cam)
