"""The painter's sort of transparent meshes around the edges of its one-block
form (powers of two, 4,096 triangles, a job with one larger mesh): after each
frame the persistent order of every mesh equals the oracle's."""
import numpy as np
import pytest

import cases
from draw_gb300 import scenes as S
from helpers import compare, describe, oracle_render
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


@pytest.mark.parametrize("frames", [1, 3, 17])
def test_sorted_beside_opaque_triangles(frames, gpu_ctx, oracle_lib):
    """Frames with opaque triangles as well, whose front runs beside the sort of a
    small job: order after each of two renders, and the first one's pixels."""
    from draw_gb300 import renderer

    sizes = (3, 700, 64)
    descs = []
    for f in range(frames):
        rng = np.random.Generator(np.random.PCG64(f))
        n = sum(sizes)
        pos = (rng.uniform(-3.0, 3.0, (n, 1, 3)) + rng.uniform(-0.5, 0.5, (n, 3, 3))).reshape(-1, 3)
        glass = cases._obj(pos, np.arange(3 * n).reshape(-1, 3), [cases._tmat(0.5, 0)],
                           mesh_split=[(s, 0) for s in sizes])
        solid = rng.uniform(-3.0, 3.0, (300, 3))
        opaque = cases._obj(solid, np.arange(300).reshape(-1, 3), [cases._mat(0)])
        descs.append(cases.flat_scene([opaque, glass], width=48 + f, height=40,
                                      textures=[S.value_noise_checker(32, 32, 5)]))
    oracles = [_oracle_objects(d) for d in descs]
    built = [renderer.build_scene(d, gpu_ctx) for d in descs]
    for turn, cam in enumerate(((0.0, 0.0, 10.0), (1.0, -2.0, 9.0))):
        for (o, s, c, _), b in zip(oracles, built):
            o.camera_op(s, 7, cam)
            b.scene.camera._op(7, *cam)
            assert o.render(s, c) == 0
        gpu_ctx.render_batch([b.scene for b in built], [b.canvas for b in built])
        gpu_ctx.synchronize()
        assert gpu_ctx.last_stats()["launches"] == 7
        for d, (o, _, _, oids), b in zip(descs, oracles, built):
            for mi, size in enumerate(sizes):
                want = o.transparent_tris(oids[1], mi, size)
                assert np.array_equal(want, b.objects[1].transparent_triangles(mi)), (d.width, mi, cam)
            if turn == 0:
                ref = oracle_render(d)
                p = compare(ref, (*b.canvas.read(), 0), d.clear_depth)
                assert p.ok and p.n_covered > 100, describe(p)
