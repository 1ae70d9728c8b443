"""The render server reserves a batch's scratch before it launches it, by the same
sizes that the launch then allocates: a request of micro triangles, whose job also
holds a survivor rest list, is admitted exactly when all of it fits the budget."""
import numpy as np
import pytest

import test_gpu_lean as lean
from draw_gb300 import scenes as S

pytestmark = pytest.mark.gpu

DG_E_OOM = 7


def _serve(budget, desc):
    """(status, peak bytes) of one request on a server of its own."""
    from draw_gb300 import renderer as R

    ctx = R.Context(0)
    try:
        maps = [R.TextureMap(t.img, t.width, t.height, t.comps, ctx) for t in desc.textures]
        ob = R.upload_object(desc.objects[0], maps, ctx)
        srv = R.Server(ctx, budget_bytes=budget, max_batch=4, streams=1)
        w, h = desc.canvas_size
        ticket = srv.submit(R.Server.request(ob, w, h, desc.cam_pos, desc.cam_dir, desc.near, desc.far, desc.fov_x,
                                             desc.lights))
        status = 0
        try:
            srv.wait(ticket)
        except R.DrawError as e:
            status = e.status
        peak = int(srv.stats()["peak_bytes"])
        srv.close()
    finally:
        ctx.close()
    return status, peak


@pytest.mark.parametrize("kind", ["micro", "ordinary"])
def test_scratch_is_reserved_whole(kind):
    if kind == "micro":
        desc = lean._micro()
    else:  # more triangles than the one-kernel front takes, so that every buffer is used
        desc = S.sphere_field(width=420, height=230, n_spheres=150, slices=50, stacks=21, tex=64, box=12.0)
        assert desc.n_tris > 131072
    desc.lights = np.asarray(desc.lights, np.float32)[:8]
    status, peak = _serve(8 << 30, desc)
    assert status == 0
    assert _serve(peak, desc) == (0, peak)
    status, less = _serve(peak - 1, desc)
    assert status == DG_E_OOM and less <= peak - 1
