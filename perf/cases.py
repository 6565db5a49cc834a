"""The work a program has this framework do, as cases that can be timed.

A case is one pass of a frame loop: clear the target, render, hand the image
to the copy stream (read_async into page-locked arrays).  Sizes and scenes
are those of this repository's benchmark (scenes.py): the fill-stress frame,
the instanced cubes, the heightfield grids of the serving set, uneven
batches and the serving mix, and ragged and small ones between them.

Kinds:
  cube    one textured cube, the smallest frame: launches and latency
  fill    clip-space triangles of log-uniform area, any shader, context
          options, optionally re-uploaded on every pass (streaming)
  grid    one heightfield mesh under an orbit camera: many small triangles
  floor   instanced cubes, one render() call each, in one pass
  crates  a first-person camera among crates with object culling
  batch   independent uneven scenes in one pass
  serve   a burst of requests through the serving loop
  lines   a grid's wireframe
"""
import math

import numpy as np
import torch

import retrofire_gb300 as rf
from retrofire_gb300 import mat, scenes

NATTR = {"flat": 0, "gouraud": 3, "textured": 2, "tex_gouraud": 5, "gouraud_srgb": 3}
# As scenes.SERVING_MESHES: the grids' edge lengths, triangles 2 n^2.
SERVE_TRIS = (12, 128, 2048, 32768, 500000)


def listed():
    return [
        # The drop-in call on the smallest scene, stats returned on every
        # call: pure latency, host path included.
        dict(name="cube_call", kind="cube", w=640, h=480, graphs=False, stats=True),
        # The same frame in a loop that replays it as a CUDA graph.
        dict(name="cube_loop", kind="cube", w=640, h=480, graphs=True, stats=False),
        # An ordinary, ragged frame: odd width, a few thousand triangles.
        dict(name="fill_7k_ragged", kind="fill", tris=7013, w=1283, h=719, shader="gouraud",
             graphs=False, stats=False, sort=0, depth=True, stream=False),
        # The benchmark frame: 1080p, 100 k Gouraud triangles, replayed.
        dict(name="fill_100k", kind="fill", tris=100000, w=1920, h=1080, shader="gouraud",
             graphs=True, stats=False, sort=0, depth=True, stream=False),
        # The same with the mesh re-submitted from host memory on every frame.
        dict(name="fill_100k_stream", kind="fill", tris=100000, w=1920, h=1080, shader="gouraud",
             graphs=True, stats=False, sort=0, depth=True, stream=True),
        # Painter's algorithm: depth-sorted triangles into a colour-only target.
        dict(name="painter_20k", kind="fill", tris=20000, w=1024, h=768, shader="gouraud",
             graphs=False, stats=False, sort=2, depth=False, stream=False),
        # Ten thousand objects, one render() call each, in one pass.
        dict(name="floor_10k", kind="floor", objects=10000, tex=1024, w=1920, h=1080, graphs=True),
        # A first-person view among crates, each tested against the frustum.
        dict(name="crates_1600", kind="crates", objects=1600, tex=256, w=1280, h=720, graphs=False),
        # The largest mesh of the serving set: half a million small triangles.
        dict(name="grid_500k", kind="grid", n=500, shader="tex_gouraud", w=1920, h=1080,
             graphs=False, stats=False),
        # Independent uneven scenes in one pass.
        dict(name="batch_64", kind="batch", scenes=64, mix=4, tris_max=200000, graphs=True),
        # A burst of 32 requests of the serving mix.
        dict(name="serve_32", kind="serve", requests=32, mix=5),
        # A wireframe: 12,416 lines.
        dict(name="wire_64", kind="lines", n=64, w=1280, h=720),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cube", "fill", "fill", "fill", "fill", "floor", "crates", "grid", "grid",
                       "batch", "serve", "lines"])
    w, h = _log(rng, 64, 1920), _log(rng, 64, 1080)
    if rng.random() < 0.5:
        w, h = rng.choice([(320, 240), (640, 480), (1280, 720), (1920, 1080)])
    loop = rng.random() < 0.5
    if kind == "cube":
        return dict(kind=kind, w=w, h=h, graphs=loop, stats=not loop)
    if kind == "fill":
        sort = rng.choice([0, 0, 0, 0, 1, 2])
        return dict(kind=kind, tris=_log(rng, 12, 200000), w=w, h=h,
                    shader=rng.choice(["flat", "gouraud", "gouraud", "gouraud_srgb"]), graphs=loop,
                    stats=rng.random() < 0.25, sort=sort, depth=sort == 0, stream=rng.random() < 0.25)
    if kind == "floor":
        return dict(kind=kind, objects=_log(rng, 50, 10000), tex=rng.choice([64, 256, 1024]), w=w, h=h,
                    graphs=loop)
    if kind == "crates":
        return dict(kind=kind, objects=_log(rng, 50, 5000), tex=rng.choice([64, 256, 1024]), w=w, h=h,
                    graphs=loop)
    if kind == "grid":
        return dict(kind=kind, n=_log(rng, 8, 500), shader=rng.choice(["gouraud", "tex_gouraud"]), w=w,
                    h=h, graphs=loop, stats=rng.random() < 0.5)
    if kind == "batch":
        return dict(kind=kind, scenes=_log(rng, 4, 64), mix=rng.randrange(1, 1000), tris_max=20000,
                    graphs=loop)
    if kind == "serve":
        return dict(kind=kind, requests=_log(rng, 4, 32), mix=rng.randrange(1, 1000))
    return dict(kind="lines", n=_log(rng, 8, 128), w=w, h=h)


# ---- inputs -----------------------------------------------------------------
# A scene: w, h, vp and draws, each (verts, faces, mvp or None for clip space).

def _seed(*parts):
    return int(np.random.SeedSequence([int(p) for p in parts]).generate_state(1)[0] >> 1) + 1


def _fill(tris, w, h, seed, shader="gouraud"):
    # The area range scales with the target's share of a 1080p frame, as in
    # scenes.batch_scenes.
    amax = max(4.0, 1e4 * (w * h) / (1920.0 * 1080.0))
    s = scenes.fill_stress(ntri=tris, w=w, h=h, seed=seed, amax=amax)
    v = np.ascontiguousarray(s["verts"][:, :4 + NATTR[shader]])
    return dict(w=w, h=h, vp=s["vp"], draws=[(v, s["faces"], None)])


def _floor(objects, tex, w, h, seed):
    s = scenes.instanced_cubes(ninst=objects, w=w, h=h, seed=seed, tex_size=tex)
    return dict(w=w, h=h, vp=s["vp"], tex=s["tex"],
                draws=[(s["verts"], s["faces"], m) for m in s["mvps"]])


def _crates(objects, tex, w, h, seed):
    """Crates on a square lattice around the camera, which stands at its
    middle, two units up, and looks along a drawn heading."""
    rng = np.random.default_rng(seed)
    side = int(math.ceil(math.sqrt(objects)))
    i = np.arange(objects)
    model = np.tile(np.eye(4, dtype=np.float32), (objects, 1, 1))
    model[:, 0, 3] = (i % side - side / 2.0) * 5.0 + rng.uniform(-1.0, 1.0, objects) + 2.5
    model[:, 1, 3] = 0.5
    model[:, 2, 3] = (i // side - side / 2.0) * 5.0 + rng.uniform(-1.0, 1.0, objects) + 2.5
    a = rng.uniform(0.0, 2.0 * math.pi)
    cam = scenes.first_person_camera([0.0, 2.0, 0.0], [math.sin(a), 1.95, math.cos(a)], w, h,
                                     lambda r: mat.focal_ratio_diagonal(np.pi / 2.0, r), 0.1, 1000.0)
    verts, faces = scenes.cube_mesh(1.0, "uv")
    mvps = mat.then(model, cam.world_to_project())
    return dict(w=w, h=h, vp=cam.viewport_m, tex=scenes.noise_texture(tex, seed),
                draws=[(verts, faces, m) for m in mvps])


def _grid(n, shader, w, h, seed):
    verts, faces = scenes.grid_mesh(n, _seed(seed, 1) % 1000, "col_uv" if shader == "tex_gouraud" else "col")
    return dict(w=w, h=h, vp=mat.viewport(0, h, w, 0), tex=scenes.noise_texture(256, seed),
                draws=[(verts, faces, scenes.orbit_camera(seed, w, h))])


def _batch(case, seed):
    """Sizes and recipes from `mix`, contents from the seed."""
    rng = np.random.default_rng(case["mix"])
    out = []
    for i in range(case["scenes"]):
        w = int(round(np.exp(rng.uniform(np.log(64), np.log(1920)))))
        h = int(round(np.exp(rng.uniform(np.log(64), np.log(1080)))))
        t = int(round(np.exp(rng.uniform(np.log(12), np.log(case["tris_max"])))))
        tex = 1 << int(rng.integers(6, 11))
        if rng.random() < 0.5:
            out.append(_fill(max(1, t), w, h, _seed(seed, i)))
        else:
            out.append(_floor(max(1, t // 12), tex, w, h, _seed(seed, i)))
    return out


def _lines(n):
    """Every distinct edge of grid_mesh(n): along x, along z, one diagonal."""
    k = np.arange((n + 1) * (n + 1)).reshape(n + 1, n + 1)
    e = [np.stack([a.reshape(-1), b.reshape(-1)], -1)
         for a, b in ((k[:, :-1], k[:, 1:]), (k[:-1], k[1:]), (k[:-1, :-1], k[1:, 1:]))]
    return np.concatenate(e).astype(np.uint32)


def _scenes(case, seed):
    k = case["kind"]
    if k == "cube":
        s = scenes.textured_cube(seed=_seed(seed), w=case["w"], h=case["h"])
        return [dict(w=s["w"], h=s["h"], vp=s["vp"], tex=s["tex"], draws=[(s["verts"], s["faces"], s["mvp"])])]
    if k == "fill":
        return [_fill(case["tris"], case["w"], case["h"], _seed(seed), case["shader"])]
    if k == "floor":
        return [_floor(case["objects"], case["tex"], case["w"], case["h"], _seed(seed))]
    if k == "crates":
        return [_crates(case["objects"], case["tex"], case["w"], case["h"], _seed(seed))]
    if k == "grid":
        return [_grid(case["n"], case["shader"], case["w"], case["h"], _seed(seed))]
    return _batch(case, seed)


def _serve_mix(case):
    """(mesh, w, h) of every request: scenes.serving_requests' mix."""
    return [(r["mesh"], r["w"], r["h"]) for r in scenes.serving_requests(case["requests"], 1000.0, seed=case["mix"])]


# ---- the program's own state ------------------------------------------------

_devices = {}
_served = {}


def _device(graphs):
    """One device context per program, as rf.default_device() is; a loop
    that replays its frames keeps one with graphs on."""
    if graphs not in _devices:
        _devices[graphs] = rf.Device()
        _devices[graphs].set_graphs(graphs)
    return _devices[graphs]


def _server():
    """The serving program: its meshes and texture are uploaded once, then
    the server takes over the context."""
    if not _served:
        dev = rf.Device()
        tex = rf.Texture(scenes.noise_texture(256, 9), device=dev)
        kinds = {"textured": rf.TEXTURED, "gouraud": rf.GOURAUD, "tex_gouraud": rf.TEX_GOURAUD}
        meshes = []
        for _, sh, build in scenes.SERVING_MESHES:
            v, f = build()
            meshes.append((rf.Mesh(v, f, device=dev), rf.Shader(kinds[sh], texture=tex if sh != "gouraud" else None)))
        _served.update(dev=dev, tex=tex, meshes=meshes, server=rf.Server(dev))
    return _served


def _pinned(n, dtype):
    return torch.empty(n, dtype=dtype, pin_memory=True)


class _State:
    """Handles and page-locked buffers of one program state."""

    def __init__(self):
        self.handles = []

    def own(self, x):
        self.handles.append(x)
        return x

    def __del__(self):
        for x in self.handles:
            x.close()


def _images(st, sizes, depth):
    """Page-locked images of every target, end to end, and views of each."""
    n = sum(w * h for w, h in sizes)
    st.keep = [_pinned(n, torch.int32)] + ([_pinned(n, torch.float32)] if depth else [])
    st.color = st.keep[0].numpy()
    st.depth = st.keep[1].numpy() if depth else None
    st.views, at = [], 0
    for w, h in sizes:
        st.views.append((st.color[at:at + w * h], st.depth[at:at + w * h] if depth else None))
        at += w * h


def prepare(case, seed):
    st = _State()
    st.case = case
    k = case["kind"]
    if k == "serve":
        s = _server()
        mix = _serve_mix(case)
        st.server = s["server"]
        st.requests = []
        _images(st, [(w, h) for _, w, h in mix], False)
        for i, (m, w, h) in enumerate(mix):
            mesh, shader = s["meshes"][m]
            st.requests.append(([(mesh, shader, scenes.orbit_camera(_seed(seed, i), w, h))],
                                mat.viewport(0, h, w, 0), w, h, st.views[i][0].reshape(h, w).view(np.uint32)))
        return st
    if k == "lines":
        dev = _device(False)
        n, w, h = case["n"], case["w"], case["h"]
        verts, _ = scenes.grid_mesh(n, _seed(seed, 1) % 1000)
        st.target = st.own(rf.Framebuf(w, h, device=dev))
        st.lines = st.own(rf.Lines(verts, _lines(n), device=dev))
        st.mvp, st.vp, st.shader = scenes.orbit_camera(_seed(seed), w, h), mat.viewport(0, h, w, 0), rf.Shader.gouraud()
        _images(st, [(w, h)], True)
        return st
    dev = st.dev = _device(case["graphs"])
    depth = case.get("depth", True)
    scs = _scenes(case, seed)
    flags = rf.DRAW_CULL_BBOX if k == "crates" else 0
    st.scenes, st.targets = [], []
    for s in scs:
        tg = st.own(rf.Framebuf(s["w"], s["h"], pixfmt=rf.ARGB8888 if depth else rf.RGBA8888, depth=depth, device=dev))
        st.targets.append(tg)
        verts, faces, mvp = s["draws"][0]
        mesh = st.own(rf.Mesh(verts, faces, pos_dim=4 if mvp is None else 3, device=dev))
        tex = st.own(rf.Texture(s["tex"], device=dev)) if "tex" in s else None
        if k in ("fill", "grid"):
            name = case["shader"]
        else:
            name = "textured" if k in ("cube", "crates") else "gouraud" if mvp is None else "tex_gouraud"
        shader = {"flat": lambda: rf.Shader.flat(0xFF4080C0), "gouraud": rf.Shader.gouraud,
                  "gouraud_srgb": rf.Shader.gouraud_srgb, "textured": lambda: rf.Shader.textured(tex),
                  "tex_gouraud": lambda: rf.Shader.tex_gouraud(tex)}[name]()
        sort = case.get("sort", 0)
        ctx = rf.Context(depth_sort=sort, depth_test=rf.DEPTH_LESS if depth else rf.DEPTH_NONE)
        st.scenes.append(rf.Scene(tg, [(mesh, shader, m, flags) for _, _, m in s["draws"]], s["vp"], ctx))
        st.mesh, st.shader, st.mvp, st.vp, st.ctx = mesh, shader, mvp, s["vp"], ctx
        if case.get("stream"):
            st.host = [torch.from_numpy(np.ascontiguousarray(verts)).pin_memory(),
                       torch.from_numpy(np.ascontiguousarray(faces).view(np.int32)).pin_memory()]
            st.host = [(st.host[0], st.host[0].numpy()), (st.host[1], st.host[1].numpy().view(np.uint32))]
    _images(st, [(s["w"], s["h"]) for s in scs], depth)
    return st


def run(st):
    k = st.case["kind"]
    if k == "serve":
        tickets = [st.server.submit(d, vp, w, h, color_out=out, read_depth=False)
                   for d, vp, w, h, out in st.requests]
        done = [st.server.wait(t) for t in tickets]
        return {"color": st.color, "frags": [r["stats"].frags_o for _, _, r in done]}
    out = {"color": st.color}
    if st.depth is not None:
        out["depth"] = st.depth
    if k == "lines":
        st.target.clear()
        s = rf.render_lines(st.lines, st.shader, st.mvp, st.vp, st.target)
        st.target.read_async(*st.views[0])
        out["stats"] = [s.prims_o, s.frags_i, s.frags_o, s.oob]
        return out
    if st.case.get("stream"):
        st.mesh.update_async(st.host[0][1], st.host[1][1])
    for tg in st.targets:
        tg.clear()
    if st.case.get("stats"):
        # The drop-in call: render() with its stats.
        s = rf.render(st.mesh, None, st.shader, st.mvp, st.vp, st.targets[0], st.ctx)
        out["stats"] = [s.prims_o, s.verts_o, s.frags_i, s.frags_o, s.oob]
    else:
        rf.render_batch(st.scenes, device=st.dev, sync_stats=False)
    for tg, (c, d) in zip(st.targets, st.views):
        tg.read_async(c, d)
    return out


# ---- what a pass cannot do without ------------------------------------------

def work(case):
    """Vertices, indices and texels in, the images out; per vertex the
    transform and outcode (28 + 42 operations), per triangle the divides,
    winding and gradients (about 150), per covered pixel one depth step and
    the colour's (2 + 4).  Covered pixels: the recipes' mean areas, and a
    third of the target for a view of a mesh."""
    k = case["kind"]

    def fill(tris, w, h, na):
        amax = max(4.0, 1e4 * (w * h) / (1920.0 * 1080.0))
        return 3 * tris, tris, 4 + na, tris * (amax - 1.0) / math.log(amax), 0

    def view(nv, nt, width, w, h, texels):
        return nv, nt, width, w * h / 3.0, texels

    if k == "batch":
        rng = np.random.default_rng(case["mix"])
        parts, px = [], 0
        for _ in range(case["scenes"]):
            w = int(round(np.exp(rng.uniform(np.log(64), np.log(1920)))))
            h = int(round(np.exp(rng.uniform(np.log(64), np.log(1080)))))
            t = int(round(np.exp(rng.uniform(np.log(12), np.log(case["tris_max"])))))
            tex = 1 << int(rng.integers(6, 11))
            px += w * h
            parts.append(fill(t, w, h, 3) if rng.random() < 0.5 else view(24 * (t // 12 + 1), t, 0, w, h, tex * tex))
        image = 8 * px
    elif k == "serve":
        mix = _serve_mix(case)
        parts = [view(SERVE_TRIS[m] // 2 + 4, SERVE_TRIS[m], 8, w, h, 0) for m, w, h in mix]
        image = sum(4 * w * h for _, w, h in mix)
    else:
        w, h = case["w"], case["h"]
        image = (8 if case.get("depth", True) else 4) * w * h
        if k == "cube":
            parts = [view(24, 12, 5, w, h, 64 * 64)]
        elif k == "fill":
            parts = [fill(case["tris"], w, h, NATTR[case["shader"]])]
        elif k == "grid":
            n = case["n"]
            parts = [view((n + 1) ** 2, 2 * n * n, 3 + NATTR[case["shader"]], w, h, 256 * 256)]
        elif k == "lines":
            n = case["n"]
            parts = [((n + 1) ** 2, n * (3 * n + 2), 6, 10.0 * n * n, 0)]
        else:  # one shared mesh, a matrix per object
            parts = [view(24 * case["objects"], 12 * case["objects"], 0, w, h, case["tex"] ** 2)]
            image += 64 * case["objects"]
    nb = sum(4 * nv * width + (12 * nt if width else 0) + 4 * tx for nv, nt, width, _, tx in parts) + image
    fl = sum(70 * nv + 150 * nt + 6 * px for nv, nt, _, px, _ in parts)
    return {"bytes": nb, "flops": fl}


# ---- the depth image in 64 bits ---------------------------------------------

def _depth64(s):
    """The depth buffer of a scene drawn with the default context on a
    cleared target: per pixel the largest 1/w of the front-facing triangles
    that cover its centre between the near and far planes.  Coverage and
    depth come from the triangle's homogeneous coordinates at the pixel
    centre, so vertices behind the eye need no clipping."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    f8 = torch.float64
    w, h = s["w"], s["h"]
    vp = torch.tensor(np.asarray(s["vp"], np.float64), device=dev)
    out = torch.zeros(w * h, dtype=f8, device=dev)
    verts0, faces, m0 = s["draws"][0]
    idx = torch.from_numpy(faces.astype(np.int64)).to(dev)
    if m0 is None:
        clip = torch.from_numpy(verts0[:, :4].astype(np.float64)).to(dev)[idx]
    else:
        p = torch.from_numpy(np.c_[verts0[:, :3], np.ones(len(verts0))].astype(np.float64)).to(dev)
        mv = torch.from_numpy(np.stack([m for _, _, m in s["draws"]]).astype(np.float64)).to(dev)
        clip = (p[None] @ mv.transpose(1, 2))[:, idx].reshape(-1, 3, 4)
    hx = vp[0, 0] * clip[..., 0] + vp[0, 3] * clip[..., 3]
    hy = vp[1, 1] * clip[..., 1] + vp[1, 3] * clip[..., 3]
    hw, hz = clip[..., 3], clip[..., 2]
    hom = torch.stack([hx, hy, hw], -1)  # (t, 3, 3): one row per vertex
    det = torch.linalg.det(hom)
    ahead = (hw > 0).any(1)
    # Bounding boxes; the whole target where a vertex lies behind the eye.
    big = (hw <= 0).any(1)
    sx, sy = torch.where(hw > 0, hx / hw, hx * 0), torch.where(hw > 0, hy / hw, hy * 0)
    x0 = torch.where(big, torch.zeros_like(det), sx.amin(1).clamp(0, w)).floor().long()
    x1 = torch.where(big, torch.full_like(det, w), sx.amax(1).clamp(0, w)).ceil().long()
    y0 = torch.where(big, torch.zeros_like(det), sy.amin(1).clamp(0, h)).floor().long()
    y1 = torch.where(big, torch.full_like(det, h), sy.amax(1).clamp(0, h)).ceil().long()
    keep = (det > 0) & ahead & (x1 > x0) & (y1 > y0)
    hom, hz, x0, x1, y0, y1 = (v[keep] for v in (hom, hz, x0, x1, y0, y1))
    inv = torch.linalg.inv(hom) if len(hom) else hom  # b = (px, py, 1) @ inv
    area = (x1 - x0) * (y1 - y0)
    ends = area.cumsum(0).cpu().numpy()
    t0 = 0
    while t0 < len(area):
        t1 = max(t0 + 1, int(np.searchsorted(ends, (ends[t0 - 1] if t0 else 0) + 8_000_000, "right")))
        n = area[t0:t1]
        t = torch.repeat_interleave(torch.arange(t0, t1, device=dev), n)
        k = torch.arange(len(t), device=dev) - torch.repeat_interleave(n.cumsum(0) - n, n)
        wd = (x1 - x0)[t]
        px, py = x0[t] + k % wd, y0[t] + k // wd
        b = [(px + 0.5) * inv[t, 0, i] + (py + 0.5) * inv[t, 1, i] + inv[t, 2, i] for i in range(3)]
        z = b[0] * hz[t, 0] + b[1] * hz[t, 1] + b[2] * hz[t, 2]
        ok = (b[0] >= 0) & (b[1] >= 0) & (b[2] >= 0) & (z.abs() <= 1.0)
        out.scatter_reduce_(0, (py * w + px)[ok], (b[0] + b[1] + b[2])[ok], "amax")
        t0 = t1
    return out.cpu().numpy()


def exact(case, seed):
    """The depth image; colours and stats are whole numbers, decided bit for
    bit by the f32 sums along every row, and have no such value."""
    if case["kind"] in ("serve", "lines") or not case.get("depth", True):
        return None
    out = {"color": None, "depth": np.concatenate([_depth64(s) for s in _scenes(case, seed)])}
    if case.get("stats"):
        out["stats"] = [None] * 5
    return out
