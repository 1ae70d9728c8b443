"""The workloads this renderer is timed on, through its public entry points.

Each case is one thing that a user of the package has it do: a frame of a
scene (Scene.render), a batch of frames (Context.render_batch, Batch.render), a
burst of requests to the render server (Server), a frame with transparent
meshes, a frame with the 2D overlay drawn over it. Sizes are those of the
package's own configurations and tests (draw_gb300/scenes.py), from a
thumbnail of a 200-triangle mesh to a 3840x2160 frame of 10 million triangles.

A case is a dict of plain values. `prepare` makes what a program holds before
the call (a context, uploaded meshes and texture maps, scenes, canvases) from
the case and a seed; `run` is one pass; its outputs are the canvases' colour
(BGRA bytes, row 0 = top) and depth (row 0 = the bottom row) buffers.
"""
import math

import numpy as np
import torch

from draw_gb300 import renderer as R
from draw_gb300 import scenes as S

_stream = None


def listed():
    """The cases, smallest first. Fields: kind (what is called), w, h (frame size),
    tris (triangles, about), tex (texture side), comps (bytes per texel), lights."""
    return [
        # A thumbnail of a small model, as an asset browser draws it: five dependent launches, no work.
        dict(name="thumbnail_96x64", kind="mesh", shape="torus", w=96, h=64, tris=200, tex=64, comps=3, lights=1,
             exponent=2),
        # The package's plain configuration: an 800x600 window (the application's default size) of one torus.
        dict(name="torus_800x600", kind="mesh", shape="torus", w=800, h=600, tris=4800, tex=512, comps=4, lights=1,
             exponent=32),
        # A finely tessellated model in a small square frame, an RGB texture and three lights.
        dict(name="sphere_512x512", kind="mesh", shape="sphere", w=512, h=512, tris=100_000, tex=1024, comps=3,
             lights=3, exponent=5),
        # Both opt-in modes (perspective-correct interpolation, bilinear fetch) at an odd frame size.
        dict(name="field_modes_1283x717", kind="field", w=1283, h=717, spheres=120, slices=40, stacks=21, tex=777,
             lights=2, modes=True),
        # The package's configuration at scale: a 1080p frame of a million triangles, some crossing the near plane.
        dict(name="field_1920x1080", kind="field", w=1920, h=1080, spheres=500, slices=50, stacks=21, tex=2048,
             lights=2, modes=False),
        # A 4K frame of ordinary geometry: large triangles, many pixels.
        dict(name="field_3840x2160", kind="field", w=3840, h=2160, spheres=160, slices=40, stacks=16, tex=2048,
             lights=1, modes=False),
        # The stress configuration: 10 million triangles of about two pixels each, four lights.
        dict(name="micro_3840x2160", kind="micro", w=3840, h=2160, tris=10_000_000, tex=4096, lights=4),
        # Uneven small frames rendered as one job, replayed from a captured graph (the batched form).
        dict(name="batch_graph_32", kind="batch", frames=32, graph=True, side_lo=128, side_hi=512, tris_lo=1_000,
             tris_hi=200_000, tex=512, mix=1234),
        # A few frames handed over in one call, without a captured graph.
        dict(name="batch_call_10", kind="batch", frames=10, graph=False, side_lo=96, side_hi=720, tris_lo=2_000,
             tris_hi=60_000, tex=256, mix=77),
        # The render server: a burst of requests of mixed sizes, every frame read back by its client.
        dict(name="serve_burst_16", kind="serve", requests=16, side_lo=128, side_hi=768, tris_lo=5_000,
             tris_hi=400_000, meshes=6, tex=512, mix=5),
        # Glass: transparent meshes (painter's sort, ordered blend) in front of an opaque model.
        dict(name="glass_1280x720", kind="glass", w=1280, h=720, tris=20_000, bubbles=24, bubble_tris=800, panes=1,
             fill=0.6, tex=512, lights=2),
        # A GUI drawn over the frame: windows and glyph quads as textured, clipped, blended 2D triangles.
        dict(name="overlay_800x600", kind="overlay", w=800, h=600, tris=4800, tex=256, lights=1, windows=6,
             glyphs=900),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _side(rng, lo, hi):
    return max(1, int(round(_log(rng, lo, hi))))


def draw(rng):
    """One more case of the same ranges: sizes spread over their logarithm, odd ones among them."""
    kind = rng.choice(["mesh", "mesh", "mesh", "field", "field", "micro", "batch", "batch", "serve", "glass", "glass",
                       "overlay", "overlay"])
    if kind == "mesh":
        w = _side(rng, 64, 1920)
        return dict(kind=kind, shape=rng.choice(["torus", "sphere"]), w=w, h=max(48, int(w * rng.uniform(0.5, 1.1))),
                    tris=_side(rng, 200, 400_000), tex=_side(rng, 32, 1024), comps=rng.choice([3, 4]),
                    lights=rng.randint(1, 4), exponent=rng.choice([1, 2, 5, 32]))
    if kind == "field":
        w = _side(rng, 320, 3840)
        return dict(kind=kind, w=w, h=max(180, int(w * rng.uniform(0.5, 0.8))), spheres=_side(rng, 20, 500),
                    slices=rng.randint(12, 50), stacks=rng.randint(8, 21), tex=_side(rng, 64, 2048),
                    lights=rng.randint(1, 4), modes=rng.random() < 0.3)
    if kind == "micro":
        w = _side(rng, 320, 2560)
        return dict(kind=kind, w=w, h=int(w * 9 / 16) | 1, tris=_side(rng, 100_000, 4_000_000),
                    tex=_side(rng, 256, 2048), lights=rng.randint(1, 4))
    if kind == "batch":
        lo, tlo = _side(rng, 64, 256), _side(rng, 500, 10_000)
        return dict(kind=kind, frames=rng.randint(2, 32), graph=rng.random() < 0.5, side_lo=lo,
                    side_hi=lo * rng.randint(2, 4), tris_lo=tlo, tris_hi=tlo * rng.randint(2, 16),
                    tex=_side(rng, 64, 512), mix=rng.randint(0, 9999))
    if kind == "serve":
        lo, tlo = _side(rng, 96, 256), _side(rng, 2_000, 20_000)
        return dict(kind=kind, requests=rng.randint(2, 24), side_lo=lo, side_hi=lo * rng.randint(2, 4), tris_lo=tlo,
                    tris_hi=tlo * rng.randint(2, 16), meshes=rng.randint(1, 8), tex=_side(rng, 64, 512),
                    mix=rng.randint(0, 9999))
    if kind == "glass":
        w = _side(rng, 160, 1920)
        return dict(kind=kind, w=w, h=max(90, int(w * rng.uniform(0.5, 0.9))), tris=_side(rng, 500, 100_000),
                    bubbles=rng.randint(1, 60), bubble_tris=_side(rng, 48, 3000), panes=rng.randint(0, 1),
                    fill=round(rng.uniform(0.1, 0.8), 3), tex=_side(rng, 32, 512), lights=rng.randint(1, 3))
    w = _side(rng, 200, 1920)
    return dict(kind=kind, w=w, h=max(120, int(w * rng.uniform(0.5, 0.9))), tris=_side(rng, 500, 20_000),
                tex=_side(rng, 64, 512), lights=rng.randint(1, 2), windows=rng.randint(1, 12),
                glyphs=_side(rng, 20, 4000))


# ------------------------------------------------------------------ inputs
def _texture(rng, side, comps, alpha=False):
    """A two-colour checkerboard shaded by coarse noise, side x side texels."""
    cells = (side + 15) // 16
    noise = rng.integers(96, 256, (cells, cells), np.uint16)
    yy, xx = np.indices((cells, cells))
    base = np.where(((xx + yy) & 1)[..., None] == 1, np.array([40, 110, 220]), np.array([230, 120, 40]))
    small = ((base * noise[..., None]) >> 8).astype(np.uint8)
    img = np.empty((side, side, comps), np.uint8)
    img[..., :3] = np.repeat(np.repeat(small, 16, 0)[:side], 16, 1)[:, :side]
    if comps == 4:
        img[..., 3] = rng.integers(0, 256, (side, side), np.uint8) if alpha else 255
    return S.TextureDesc(img.reshape(-1), side, side, comps)


def _material(alpha=1.0):
    return S.Material((0.1,) * 3, (0.7,) * 3, (0.2,) * 3, alpha, 0, 0)


def _orbit(rng):
    """A camera on an orbit around the origin (distance 2.6 to 4) and a light near it."""
    az, el, dist = rng.uniform(0, 2 * math.pi), rng.uniform(0.2, 1.0), rng.uniform(2.6, 4.0)
    cam = (dist * math.cos(el) * math.sin(az), dist * math.sin(el), dist * math.cos(el) * math.cos(az))
    return cam, (3.0 * math.sin(az + 1), 4.0, 3.0 * math.cos(az + 1))


def _lights(rng, n):
    return rng.uniform(-6.0, 6.0, (n, 3)).astype(np.float32) + np.array([0.0, 3.0, 0.0], np.float32)


def _mesh_desc(case, rng):
    """One textured mesh seen from an orbiting camera."""
    pos, nrm, uv, tri = S.mesh_for_tris(case.get("shape", "torus"), case["tris"])
    obj = S.ObjectDesc(pos, nrm, uv, [S.MeshDesc(S._tris9(tri), 0)], [_material()])
    cam, _ = _orbit(rng)
    return S.SceneDesc(case["w"], case["h"], cam_pos=cam, cam_dir=tuple(-c for c in cam), near=-0.5, far=-100.0,
                       fov_x=60.0, lights=_lights(rng, case["lights"]), exponent=case.get("exponent", 2),
                       textures=[_texture(rng, case["tex"], case.get("comps", 4))], objects=[obj])


def _field_desc(case, rng):
    """Seeded spheres around the camera, several of them crossing the near plane."""
    d = S.sphere_field(width=case["w"], height=case["h"], n_spheres=case["spheres"], slices=case["slices"],
                       stacks=case["stacks"], seed=int(rng.integers(1 << 30)), tex=2, n_lights=case["lights"])
    d.textures = [_texture(rng, case["tex"], 4)]
    if case["modes"]:
        d.interpolation, d.textures[0].filter = R.INTERP_PERSPECTIVE, R.FILTER_BILINEAR
    return d


def _micro_desc(case, rng):
    """Seeded micro spheres: about two pixels per triangle, depth complexity about eight."""
    d = S.micro_sphere_field(width=case["w"], height=case["h"], n_tris=case["tris"], n_lights=case["lights"],
                             seed=int(rng.integers(1 << 30)), tex=2)
    d.textures = [_texture(rng, case["tex"], 4)]
    return d


def _glass_desc(case, rng):
    """An opaque mesh behind transparent bubbles (each a closed sphere: two layers)
    and panes (half the frame each). `fill` is the bubbles' share of the frame's area."""
    d = _mesh_desc(case, rng)
    w, h = case["w"], case["h"]
    focal = w / 2 / math.tan(math.radians(30.0))
    cam = np.array(d.cam_pos)
    fwd = -cam / np.linalg.norm(cam)
    right = np.cross(fwd, [0.0, 1.0, 0.0])
    right /= np.linalg.norm(right)
    up = np.cross(right, fwd)

    def at(px, py, dist):  # the world position `dist` ahead whose projection is (px, py) pixels off centre
        return cam + dist * (fwd + px / focal * right + py / focal * up)

    base = S.mesh_for_tris("sphere", case["bubble_tris"])
    radius_px = math.sqrt(case["fill"] * w * h / 2 / math.pi / case["bubbles"])
    mats = [_material(a) for a in (0.35, 0.6, 0.8)]
    pos, nrm, uv, meshes = [], [], [], []
    for b in range(case["bubbles"]):
        dist = rng.uniform(0.9, 2.0)
        c = at(rng.uniform(-0.4, 0.4) * w, rng.uniform(-0.4, 0.4) * h, dist)
        tri = base[3] + len(base[0]) * b
        pos.append((base[0] * (radius_px * dist / focal) + c).astype(np.float32))
        nrm.append(base[1])
        uv.append(base[2])
        meshes.append(S.MeshDesc(S._tris9(tri.astype(np.uint32)), b % 3))
    n = len(base[0]) * case["bubbles"]
    for p in range(case["panes"]):
        x0, x1, dist = -0.45 * w, 0.05 * w, 0.8
        pos.append(np.array([at(x, y, dist) for x, y in ((x0, -0.4 * h), (x1, -0.4 * h), (x1, 0.4 * h),
                                                        (x0, 0.4 * h))], np.float32))
        nrm.append(np.tile(-fwd.astype(np.float32), (4, 1)))
        uv.append(np.array([[0, 0, 0], [0.9, 0, 0], [0.9, 0.9, 0], [0, 0.9, 0]], np.float32))
        meshes.append(S.MeshDesc(S._tris9(np.array([[0, 1, 2], [0, 2, 3]], np.uint32) + np.uint32(n + 4 * p)), 0))
    d.objects.append(S.ObjectDesc(np.concatenate(pos), np.concatenate(nrm), np.concatenate(uv), meshes, mats))
    return d


def _gui(case, rng):
    """A GUI's draw list: window rectangles and rows of glyph quads inside them, two
    triangles each, with the window's rectangle as the clipping rectangle."""
    w, h = case["w"], case["h"]
    per = -(-case["glyphs"] // case["windows"])
    quads, clips, left = [], [], case["glyphs"]
    for _ in range(case["windows"]):
        ww, wh = int(rng.uniform(0.2, 0.45) * w), int(rng.uniform(0.2, 0.45) * h)
        x, y = int(rng.integers(0, w - ww)), int(rng.integers(0, h - wh))
        clip = (x, y, x + ww - 1, y + wh - 1)
        quads.append((x, y, x + ww - 1, y + wh - 1, 0.0, 0.0, 0.01, 0.01, rng.integers(20, 90, 3), 0.8))
        clips.append(clip)
        cols = max(1, (ww - 8) // 9)
        for g in range(min(per, left)):
            gx, gy = x + 4 + 9 * (g % cols), y + 4 + 14 * (g // cols)
            u, v = rng.integers(0, 12, 2) / 13.0
            quads.append((gx, gy, gx + 8, gy + 13, u, v, u + 0.07, v + 0.07, rng.integers(150, 256, 3), 1.0))
            clips.append(clip)
        left -= min(per, left)
    verts = np.zeros((len(quads), 2, 3, 8), np.float32)
    for i, (x0, y0, x1, y1, u0, v0, u1, v1, rgb, alpha) in enumerate(quads):
        corner = [(x0, y0, u0, v0), (x1, y0, u1, v0), (x1, y1, u1, v1), (x0, y1, u0, v1)]
        for t, ids in enumerate(((0, 1, 2), (0, 2, 3))):
            for k, c in enumerate(ids):
                verts[i, t, k] = (*corner[c], *rgb, alpha)
    return verts.reshape(-1, 3, 8), np.repeat(np.array(clips, np.uint64), 2, 0)


def _mix(case, n):
    """The sizes of a batch's frames or a burst's requests: (side, triangles, shape), fixed by the case."""
    rng = np.random.default_rng(case["mix"])
    return [(int(round(_log(rng, case["side_lo"], case["side_hi"]))),
             int(round(_log(rng, case["tris_lo"], case["tris_hi"]))),
             ("torus", "sphere")[int(rng.integers(2))]) for _ in range(n)]


_DESCS = dict(mesh=_mesh_desc, field=_field_desc, micro=_micro_desc, glass=_glass_desc, overlay=_mesh_desc)


class _Buffer:
    """Device memory of the context as an array (no copy)."""

    def __init__(self, ptr, shape, typestr, owner):
        self.__cuda_array_interface__ = dict(data=(ptr, False), shape=shape, typestr=typestr, version=2)
        self.owner = owner


def _tensors(canvas):
    """The canvas's colour and depth buffers as tensors."""
    colour, depth = R.ctypes.c_void_p(), R.ctypes.c_void_p()
    st = canvas.ctx.lib.dg_canvas_device_ptrs(canvas.ctx.h, canvas.id, R.ctypes.byref(colour), R.ctypes.byref(depth))
    if st:
        raise R.DrawError(st, "device_ptrs")
    h, w = canvas.height, canvas.width
    return (torch.as_tensor(_Buffer(colour.value, (h, w, 4), "|u1", canvas), device="cuda"),
            torch.as_tensor(_Buffer(depth.value, (h, w), "<f4", canvas), device="cuda"))


def _context():
    """A context on the process's render stream (one stream for all of them, as one program's frames have)."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    ctx = R.Context(torch.cuda.current_device())
    ctx.set_stream(_stream.cuda_stream)
    return ctx


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    ctx = _context()
    if kind in _DESCS:
        built = R.build_scene(_DESCS[kind](case, rng), ctx)
        state = dict(kind=kind, ctx=ctx, built=built, out=_tensors(built.canvas))
        if kind == "overlay":
            t = _texture(rng, case["tex"], 4, alpha=True)
            state["atlas"] = R.TextureMap(t.img, t.width, t.height, t.comps, ctx)
            state["verts"], state["clips"] = _gui(case, rng)
        return state
    if kind == "batch":
        built = []
        for side, tris, shape in _mix(case, case["frames"]):
            built.append(R.build_scene(_mesh_desc(dict(shape=shape, w=side, h=side, tris=tris, tex=case["tex"],
                                                       lights=1), rng), ctx))
        scenes, canvases = [b.scene for b in built], [b.canvas for b in built]
        state = dict(kind=kind, ctx=ctx, built=built, scenes=scenes, canvases=canvases,
                     out=[_tensors(c) for c in canvases])
        if case["graph"]:
            state["batch"] = ctx.batch(scenes, canvases)
        return state
    # serve: a resident pool of meshes and a list of requests for them
    maps, objects = [], []
    for _, tris, shape in _mix(case, case["meshes"]):
        t = _texture(rng, case["tex"], 4)
        maps.append(R.TextureMap(t.img, t.width, t.height, t.comps, ctx))
        pos, nrm, uv, tri = S.mesh_for_tris(shape, tris)
        objects.append(R.upload_object(S.ObjectDesc(pos, nrm, uv, [S.MeshDesc(S._tris9(tri), 0)], [_material()]),
                                       [maps[-1]], ctx))
    requests = []
    for i, (side, _, _) in enumerate(_mix(case, case["requests"])):
        cam, light = _orbit(rng)
        requests.append((R.Server.request(objects[i % len(objects)], side, side, cam, tuple(-c for c in cam), -0.5,
                                          -100.0, 60.0, [light]), side))
    server = R.Server(ctx, budget_bytes=4 << 30, max_batch=32, streams=3)
    return dict(kind=kind, ctx=ctx, maps=maps, objects=objects, requests=requests, server=server)


def run(state):
    kind = state["kind"]
    if kind == "serve":
        server = state["server"]
        tickets = [(server.submit(r), side) for r, side in state["requests"]]
        return [server.wait(t, side, side, read=True)[:2] for t, side in tickets]
    if kind == "batch":
        if "batch" in state:
            state["batch"].render()
        else:
            state["ctx"].render_batch(state["scenes"], state["canvases"])
        return state["out"]
    built = state["built"]
    built.scene.render(built.canvas)
    if kind == "overlay":
        built.canvas.draw_triangles(state["verts"], state["atlas"], state["clips"])
    return state["out"]


# -------------------------------------------------------------------- work
def _frame_work(vertices, tris, px, texels):
    """Each vertex (position, normal, texture coordinate), triangle (nine indices) and
    texel read once, each pixel's colour and depth written once; six plane tests, a
    projection and a distance per vertex, a normal and three edges per triangle."""
    return 32.0 * vertices + 36.0 * tris + 4.0 * texels + 8.0 * px, 64.0 * vertices + 50.0 * tris


def work(case):
    kind = case["kind"]
    parts = []
    if kind in ("batch", "serve"):
        frames = _mix(case, case["frames" if kind == "batch" else "requests"])
        meshes = frames if kind == "batch" else _mix(case, case["meshes"])
        for i, (side, _, _) in enumerate(frames):
            tris = meshes[i % len(meshes)][1]
            parts.append(_frame_work(0.5 * tris, tris, side * side, case["tex"] ** 2))
    else:
        px, texels = case["w"] * case["h"], case["tex"] ** 2
        if kind == "field":
            tris = case["spheres"] * 2 * case["slices"] * (case["stacks"] - 1)
            vertices = case["spheres"] * (case["slices"] + 1) * (case["stacks"] + 1)
        else:
            tris = case["tris"] + (case["bubbles"] * case["bubble_tris"] if kind == "glass" else 0)
            vertices = (0.9 if kind == "micro" else 0.5) * tris
        parts.append(_frame_work(vertices, tris, px, texels))
        if kind == "overlay":  # the draw list read once
            parts.append((2 * (case["windows"] + case["glyphs"]) * (96.0 + 32.0) + 4.0 * texels, 0.0))
    return dict(bytes=sum(b for b, _ in parts), flops=sum(f for _, f in parts))


# ------------------------------------------------------------------- exact
def _matrix32(d):
    """The scene's projection (viewport * orthographic * perspective * view) in f32, as
    the pixel grid is defined on the f32 projected and rounded vertex positions."""
    f = np.float32
    norm = lambda v: np.sqrt(f(f(v[0] * v[0] + v[1] * v[1]) + v[2] * v[2]))  # noqa: E731
    cross = lambda a, b: np.array([a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2],  # noqa: E731
                                   a[0] * b[1] - a[1] * b[0]], f)
    g = np.array(d.cam_dir, f)
    g = g / norm(g)
    w = (g / norm(g)) * f(-1)
    u = cross(np.array([0, 1, 0], f), w)
    u = u / norm(u)
    v = cross(w, u)
    view = np.zeros((4, 4), f)
    for i, a in enumerate((u, v, w)):
        view[i, :3] = a / norm(a)
    view[3, 3] = 1
    tr = np.eye(4, dtype=f)
    tr[:3, 3] = -np.array(d.cam_pos, f)
    n, fa = f(d.near), f(d.far)
    r = abs(n) * np.tan(f(d.fov_x) * f(math.pi / 180) / f(2))
    t = (f(1) / f(d.ratio)) * r
    persp, orth, vp = (np.zeros((4, 4), f) for _ in range(3))
    persp[0, 0] = persp[1, 1] = n
    persp[2, 2], persp[2, 3], persp[3, 2] = n + fa, -(n * fa), 1
    orth[0, 0], orth[1, 1], orth[2, 2], orth[3, 3] = f(2) / (r + r), f(2) / (t + t), f(2) / (n - fa), 1
    orth[2, 3] = -(n + fa) / (n - fa)
    vp[0, 0], vp[0, 3], vp[1, 1], vp[1, 3] = (f(d.width) / 2, (f(d.width) - 1) / 2, f(d.height) / 2,
                                              (f(d.height) - 1) / 2)
    vp[2, 2] = vp[3, 3] = 1

    def mul(a, b):
        out = np.zeros((4, 4), f)
        for k in range(4):
            out = (out + (a[:, k:k + 1] * b[k:k + 1, :]).astype(f)).astype(f)
        return out

    return mul(mul(mul(vp, orth), persp), mul(view, tr))


def _exact_depth(d):
    """The depth buffer of the scene's first mesh (opaque, no vertex near the clipping
    planes) in 64 bits: the distance from the camera, interpolated over each
    front-facing triangle's pixels with the barycentrics of its rounded corners."""
    f = np.float32
    M, o = _matrix32(d), d.objects[0]
    p, tri = np.asarray(o.vertices, f), o.meshes[0].tris[:, :3].astype(np.int64)
    rows = [((M[i, 0] * p[:, 0] + M[i, 1] * p[:, 1]) + M[i, 2] * p[:, 2]) + M[i, 3] for i in (0, 1, 3)]
    x, y = (np.floor(rows[k] / rows[2] + f(0.5)).astype(np.float64) for k in (0, 1))
    dist = np.linalg.norm(p.astype(np.float64) - np.array(d.cam_pos, f).astype(np.float64), axis=1)
    a, b, c = (p[tri[:, k]] for k in range(3))
    e0, e1 = b - a, c - b
    nrm = np.stack([e0[:, 1] * e1[:, 2] - e0[:, 2] * e1[:, 1], e0[:, 2] * e1[:, 0] - e0[:, 0] * e1[:, 2],
                    e0[:, 0] * e1[:, 1] - e0[:, 1] * e1[:, 0]], 1)
    to = np.array(d.cam_pos, f) - ((a + b) + c) / f(3)
    tri = tri[((to[:, 0] * nrm[:, 0] + to[:, 1] * nrm[:, 1]) + to[:, 2] * nrm[:, 2]) > 0]
    w, h = d.canvas_size
    X, Y, Z = x[tri], y[tri], dist[tri]
    clamp = lambda v, n: np.clip(v, 0, n - 1).astype(np.int64)  # noqa: E731
    x0, x1, y0, y1 = clamp(X.min(1), w), clamp(X.max(1), w), clamp(Y.min(1), h), clamp(Y.max(1), h)
    count = (x1 - x0 + 1) * (y1 - y0 + 1)
    order = np.arange(len(tri))
    best = np.full(w * h, np.inf)
    edge = lambda i, px, py, k, q: ((Y[i, k] - Y[i, q]) * px + (X[i, q] - X[i, k]) * py  # noqa: E731
                                    + X[i, k] * Y[i, q] - X[i, q] * Y[i, k])
    den = np.stack([edge(order, X[:, k], Y[:, k], (k + 1) % 3, (k + 2) % 3) for k in range(3)], 1)
    tie = np.stack([den[:, k] * edge(order, -1.0, -1.0, (k + 1) % 3, (k + 2) % 3) > 0 for k in range(3)], 1)
    ends = np.cumsum(count)
    first = 0
    while first < len(tri):  # about four million pixels at a time
        last = max(first + 1, int(np.searchsorted(ends, (ends[first - 1] if first else 0) + (1 << 22), "right")))
        cnt = count[first:last]
        i = np.repeat(order[first:last], cnt)
        k = np.arange(len(i)) - np.repeat(np.cumsum(cnt) - cnt, cnt)
        bw = (x1 - x0 + 1)[i]
        px, py = x0[i] + k % bw, y0[i] + k // bw
        ok, z = np.ones(len(i), bool), np.zeros(len(i))
        with np.errstate(divide="ignore", invalid="ignore"):
            for q in range(3):
                wt = edge(i, px, py, (q + 1) % 3, (q + 2) % 3) / den[i, q]
                ok &= (wt > 0) | ((wt == 0) & tie[i, q])
                z = z + wt * Z[i, q]
        np.minimum.at(best, (py * w + px)[ok], z[ok])
        first = last
    return torch.from_numpy(best.reshape(h, w))


def exact(case, seed):
    """The depth buffer in 64 bits where one unclipped opaque mesh makes it; colours are whole bytes."""
    kind = case["kind"]
    if kind not in ("mesh", "overlay", "glass") or case["tris"] > 150_000:
        return None
    return None, _exact_depth(_DESCS[kind](case, np.random.default_rng(seed)))
