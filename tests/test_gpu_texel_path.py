"""The nearest texel fetch where its short path ends: texture coordinates that are
NaN, negative, 0, 1 and beyond the map, and maps of 1 to 4 components (with fewer
than three, the last texels' three bytes pass the end of the map). The frame, or
the texture-range status, equals the CPU oracle's."""
import numpy as np
import pytest

import cases
from draw_gb300 import scenes as S
from helpers import compare, describe, first_mismatch, gpu_render, oracle_render

pytestmark = pytest.mark.gpu

NAN = float("nan")
UVS = {
    "corners": [(0.0, 0.0), (1.0, 0.0), (1.0, 1.0), (0.0, 1.0)],
    "inside": [(0.1, 0.2), (0.93, 0.15), (0.97, 0.95), (0.02, 0.99)],
    "negative": [(-0.4, -0.2), (0.9, -0.3), (0.8, 0.9), (-0.1, 0.7)],
    "nan_u": [(NAN, 0.1), (0.5, 0.2), (0.9, 0.8), (0.1, 0.9)],
    "nan_v": [(0.2, 0.1), (0.5, NAN), (0.9, 0.8), (0.1, 0.9)],
    "u_beyond": [(0.5, 0.3), (1.6, 0.3), (1.6, 0.8), (0.5, 0.8)],
    "v_beyond": [(0.5, 0.3), (0.9, 0.3), (0.9, 1.8), (0.5, 1.8)],
    "infinite": [(0.5, 0.3), (float("inf"), 0.3), (0.9, 0.8), (0.5, 0.8)],
}


@pytest.mark.parametrize("comps", [1, 2, 3, 4])
@pytest.mark.parametrize("name", sorted(UVS))
def test_texel_path(name, comps, gpu_ctx, oracle_lib):
    rng = np.random.default_rng(comps)
    w, h = 13, 9
    tex = S.TextureDesc(rng.integers(0, 256, w * h * comps, np.uint8), w, h, comps)
    pos, tris = cases._quads([(-3.0, -2.0, 3.0, 2.0, 0.0)])
    uv = np.array([(u, v, 0.0) for u, v in UVS[name]], np.float32)
    desc = cases.flat_scene([cases._obj(pos, tris, [cases._mat(0)], uvs=uv)], textures=[tex])
    ref, got = oracle_render(desc), gpu_render(desc, gpu_ctx)
    assert ref[2] == got[2], (name, comps, ref[2], got[2])
    if ref[2] == 0:
        p = compare(ref, got, desc.clear_depth)
        assert p.ok and p.n_covered > 0, f"{describe(p)}; {first_mismatch(ref, got)}"
