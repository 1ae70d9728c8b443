"""Replays of captured batches through the paths whose kernels read counters of the
job itself: strips or whole tiles by the number of reached cells, on both sides of
the threshold in turn, and micro triangles with their survivor rest list; and the
painter's sort of a job with one large transparent mesh behind the one-kernel
front, in turn with a job of small meshes. Against the CPU oracle."""
import numpy as np
import pytest

import cases
from draw_gb300 import scenes as S
from helpers import compare, describe, first_mismatch, oracle_render
from test_gpu_lean import _micro
from test_gpu_transparent import _oracle_objects

pytestmark = pytest.mark.gpu


def _at(desc, cam):
    desc.cam_pos = tuple(float(np.float32(v)) for v in cam)
    return desc


def _replay(descs, cameras, ctx):
    """One batch of the scenes, replayed with each list of camera positions in turn."""
    from draw_gb300 import renderer

    built = [renderer.build_scene(d(), ctx) for d in descs]
    batch = ctx.batch([b.scene for b in built], [b.canvas for b in built])
    try:
        for turn, cams in enumerate(cameras):
            for b, cam in zip(built, cams):
                b.scene.camera._op(7, *cam)
            batch.render()
            for d, b, cam in zip(descs, built, cams):
                desc = _at(d(), cam)
                ref, got = oracle_render(desc), (*b.canvas.read(), 0)
                p = compare(ref, got, desc.clear_depth)
                assert p.ok and p.n_covered > 0, f"replay {turn}: {describe(p)}; {first_mismatch(ref, got)}"
        assert batch.info()["captures"] == 1
    finally:
        batch.close()


def test_strips_in_a_replay(gpu_ctx, oracle_lib):
    def torus():
        return S.torus_scene(width=1280, height=720, nu=30, nv=12, tex=64, cam_dist=3.0)

    base = np.array(torus().cam_pos)
    near, far = tuple(base * 0.8), tuple(base * 2.2)  # some 750 and 190 of 920 cells
    _replay([torus], [[far], [near], [near], [far], [far], [near]], gpu_ctx)


def test_micro_triangles_in_a_replay(gpu_ctx, oracle_lib):
    def torus():
        return S.torus_scene(width=200, height=150, nu=20, nv=10, tex=64, cam_dist=3.0)

    home = tuple(torus().cam_pos)
    moves = [(0.0, 0.0, 0.0), (0.05, 0.02, 0.0), (0.0, 0.0, 0.0), (0.1, -0.1, 0.1)]
    _replay([_micro, torus], [[m, tuple(np.array(home) + np.array(m))] for m in moves], gpu_ctx)


def _glass(sizes, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    n = sum(sizes)
    pos = (rng.uniform(-3.0, 3.0, (n, 1, 3)) + rng.uniform(-0.05, 0.05, (n, 3, 3))).reshape(-1, 3)
    glass = cases._obj(pos, np.arange(3 * n).reshape(-1, 3), [cases._tmat(0.5, 0)], mesh_split=[(s, 0) for s in sizes])
    solid = rng.uniform(-3.0, 3.0, (300, 3))
    opaque = cases._obj(solid, np.arange(300).reshape(-1, 3), [cases._mat(0)])
    return cases.flat_scene([opaque, glass], width=64, height=48, textures=[S.value_noise_checker(32, 32, 5)])


def test_large_transparent_mesh_behind_the_front(oracle_lib):
    from draw_gb300 import renderer

    ctx = renderer.Context(0)  # its first transparent job needs no sort buffers
    try:
        jobs = []
        for sizes in ((3, 700, 64), (5, 4097, 100)):
            desc = _glass(sizes, sum(sizes))
            jobs.append((sizes, desc, _oracle_objects(desc), renderer.build_scene(desc, ctx)))
        for turn, cam in enumerate(((0.0, 0.0, 10.0), (1.0, -2.0, 9.0), (0.0, 0.0, 10.0))):
            for sizes, desc, (o, s, c, oids), b in jobs:
                o.camera_op(s, 7, cam)
                b.scene.camera._op(7, *cam)
                assert o.render(s, c) == 0
                b.scene.render(b.canvas)
                ctx.synchronize()
                for mi, size in enumerate(sizes):
                    want = o.transparent_tris(oids[1], mi, size)
                    assert np.array_equal(want, b.objects[1].transparent_triangles(mi)), (sizes, mi, turn)
                if turn == 0:
                    ref, got = oracle_render(desc), (*b.canvas.read(), 0)
                    p = compare(ref, got, desc.clear_depth)
                    assert p.ok and p.n_covered > 100, f"{sizes}: {describe(p)}; {first_mismatch(ref, got)}"
    finally:
        ctx.close()
