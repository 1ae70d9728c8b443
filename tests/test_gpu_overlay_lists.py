"""The 2D overlay at the sizes where its work items and per-pixel lists change
path: a single triangle, boxes of one pixel and of more than a million pixels
(more than four units per item), stacks up to and beyond the eight fragments
that the fold orders in registers, and calls that follow one another without a
wait. Against the CPU oracle drawing the same triangles in order."""
import numpy as np
import pytest

import cases
from draw_gb300 import scenes as S
from helpers import compare, describe

pytestmark = pytest.mark.gpu


def _stack(n, w, h, seed):
    """n triangles of random corners within w x h pixels."""
    rng = np.random.default_rng(seed)
    v = np.zeros((n, 3, 8), np.float32)
    v[..., 0] = rng.uniform(-3, w + 3, (n, 3))
    v[..., 1] = rng.uniform(-3, h + 3, (n, 3))
    v[..., 2:4] = rng.uniform(0.0, 0.999, (n, 3, 2))
    v[..., 4:7] = rng.integers(0, 256, (n, 3, 3))
    v[..., 7] = rng.uniform(0.1, 1.1, (n, 3))
    return v


CASES = {
    # name: (canvas, calls as (triangles, extent))
    "one": ((64, 48), [(1, (60, 40))]),
    "one_pixel": ((1, 1), [(3, (1, 1))]),
    "stack_8": ((64, 48), [(8, (12, 12))]),
    "stack_300": ((64, 48), [(300, (10, 10))]),
    "wide_box": ((2048, 1040), [(2, (2046, 1038)), (5, (40, 40))]),
    "calls": ((200, 100), [(40, (200, 100)), (7, (30, 30)), (120, (200, 100)), (1, (9, 9)), (60, (200, 90)),
                           (33, (150, 100))]),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_overlay_lists(name, gpu_ctx, oracle_lib):
    import oracle

    from draw_gb300 import renderer

    (w, h), calls = CASES[name]
    tex = S.value_noise_checker(48, 40, 77, comps=4)
    img = tex.img.reshape(-1, 4).copy()
    img[:, 3] = np.random.default_rng(1).integers(0, 256, img.shape[0])
    batches = [_stack(n, *ext, seed=i) for i, (n, ext) in enumerate(calls)]

    o = oracle.Oracle()
    tm = o.texmap(img.reshape(-1), tex.width, tex.height, 4)
    c = o.canvas(w, h)
    o.init_depth(c, 5.0)
    for v in batches:
        for t in v:
            assert o.draw_triangle_2d(c, t, tm, None) == 0
    ref = o.read(c, w, h)

    gtm = renderer.TextureMap(img.reshape(-1), tex.width, tex.height, 4, gpu_ctx)
    canvas = renderer.Canvas(w, h, gpu_ctx)
    canvas.init_depth(5.0)
    for v in batches:
        buf = v.copy()
        canvas.draw_triangles(buf, gtm)
        buf[:] = np.nan  # the call has taken the caller's triangles
    got = canvas.read()
    p = compare((ref.bgra, ref.depth, 0), (*got, 0), 5.0)
    assert p.ok and p.colour_max_lsb == 0, describe(p)
