"""The transparent pass's per-pixel fragment lists and its painter's sort at the
sizes where they change path: lists up to and beyond the eight fragments that the
fold orders in registers, boxes whose work items one lane or the whole warp
writes, the fragment limit of a frame, and meshes around the power-of-two and
4,096-triangle edges of the one-block sort. Against the CPU oracle: depth
bit-exact, colour within 1 LSB, the persistent triangle order equal."""
import numpy as np
import pytest

import cases
from draw_gb300 import scenes as S
from helpers import compare, describe, first_mismatch, gpu_render, oracle_render

pytestmark = pytest.mark.gpu

DG_E_LIMIT = 8


def _layers(n, half, width=64, height=48, seed=3):
    """n transparent quads (half-size `half`) facing the camera at distinct depths, in
    random submission order over two meshes, and an opaque quad between them."""
    rng = np.random.Generator(np.random.PCG64(seed))
    z = np.linspace(-4.0, 4.0, n) if n > 1 else np.array([1.0])
    rng.shuffle(z)
    pos, tris = cases._quads([(-half, -half, half, half, float(v)) for v in z])
    split = [(2 * (n // 2), 0), (2 * (n - n // 2), 1)] if n > 1 else [(2, 0)]
    tr = cases._obj(pos, tris, [cases._tmat(0.5, 0), cases._tmat(0.25, 0)], mesh_split=split)
    bp, bt = cases._quads([(-1.0, -1.0, 2.0, 1.5, 0.1)])
    return cases.flat_scene([cases._obj(bp, bt, [cases._mat(0)]), tr], width=width, height=height,
                            textures=[S.value_noise_checker(32, 32, 5)])


@pytest.mark.parametrize("n", [1, 7, 8, 9, 17, 200])
def test_list_lengths(n, gpu_ctx, oracle_lib):
    desc = _layers(n, 1.5)
    ref, got = oracle_render(desc), gpu_render(desc, gpu_ctx)
    assert ref[2] == 0 and got[2] == 0
    p = compare(ref, got, desc.clear_depth)
    assert p.ok, f"{describe(p)}; {first_mismatch(ref, got)}"


@pytest.mark.parametrize("width,height", [(1, 1), (31, 5), (129, 33), (640, 360)])
def test_box_sizes(width, height, gpu_ctx, oracle_lib):
    desc = _layers(2, 30.0, width, height)
    ref, got = oracle_render(desc, frames=2), gpu_render(desc, gpu_ctx, frames=2)
    assert ref[2] == 0 and got[2] == 0
    p = compare(ref, got, desc.clear_depth)
    assert p.ok, f"{describe(p)}; {first_mismatch(ref, got)}"


def test_fragment_limit(gpu_ctx, oracle_lib):
    """A frame may have 2 x pixels + 65,536 transparent fragments: 23 full-frame layers
    of 64x48 pixels fit, 24 do not, and the frame after a refused one is unharmed."""
    fits, over = _layers(23, 30.0), _layers(24, 30.0)
    for o in (fits, over):
        o.objects.pop(0)  # the transparent layers alone
    assert gpu_render(over, gpu_ctx)[2] == DG_E_LIMIT
    ref, got = oracle_render(fits), gpu_render(fits, gpu_ctx)
    assert ref[2] == 0 and got[2] == 0
    p = compare(ref, got, fits.clear_depth)
    assert p.ok, f"{describe(p)}; {first_mismatch(ref, got)}"
    assert int((ref[0][..., 3] == 0).sum()) == 64 * 48
