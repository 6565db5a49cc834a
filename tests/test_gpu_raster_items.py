"""The rasteriser's ways of giving scanlines to lanes, against the oracle bit
for bit: triangles of few rows (32 scanlines packed to a pass), of about ten
(the line between the two ways) and of many (a lane per row), spans from one
pixel to across many tiles, coincident triangles (ties, and scanlines of one
row that wait for each other), clipped fans among them; the walk over the tile
masks when the triangle lists do not fit; jobs of every raster group in one
batch."""
import numpy as np
import pytest

import retrofire_gb300 as rf
from retrofire_gb300 import mat, scenes
from rfhelp import DrawSpec, assert_parity, gpu_render, oracle_render

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    from retrofire_gb300 import build
    build.build()
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")


NATTR = {rf.FLAT: 0, rf.GOURAUD: 3, rf.TEXTURED: 2, rf.TEX_GOURAUD: 5, rf.GOURAUD_SRGB: 3}


def tris(seed, n, w, h, size, kind=rf.GOURAUD, repeat=1, cross=0.0):
    """n clip-space triangles inside boxes of size = (xmin, xmax, ymin, ymax)
    px at random places, each repeated; a share crossing the near plane."""
    rng = np.random.default_rng(seed)
    x0, x1, y0, y1 = size
    c = rng.uniform([0, 0], [w, h], (n, 2))
    e = np.stack([rng.uniform(x0, x1, n), rng.uniform(y0, y1, n)], 1)
    px = c[:, None, :] + rng.uniform(-0.5, 0.5, (n, 3, 2)) * e[:, None, :]
    px = np.repeat(px, repeat, 0)
    n *= repeat
    wv = rng.uniform(1.0, 3.0, (n, 3))
    z = rng.uniform(-0.9, 0.9, (n, 3))
    z[rng.random(n) < cross, 0] = -1.4
    clip = np.stack([(px[..., 0] / (w / 2.0) - 1.0) * wv, (px[..., 1] / (h / 2.0) - 1.0) * wv, z * wv, wv], -1)
    verts = np.concatenate([clip, rng.uniform(0.0, 1.0, (n, 3, NATTR[kind]))], -1)
    verts = verts.reshape(3 * n, -1).astype(np.float32)
    tex = scenes.noise_texture(64, seed) if kind in (rf.TEXTURED, rf.TEX_GOURAUD) else None
    return DrawSpec(verts, np.arange(3 * n, dtype=np.uint32).reshape(n, 3), kind, pos_dim=4,
                    flat_rgba=0xFF336699, tex=tex)


SHAPES = {
    "dots": dict(n=3000, size=(1, 3, 1, 3)),
    "slivers": dict(n=1500, size=(8, 40, 1, 3)),
    "ribbons": dict(n=400, size=(150, 600, 1, 6)),
    "ten_rows": dict(n=1200, size=(4, 30, 9, 24)),
    "tall": dict(n=200, size=(2, 12, 60, 200)),
    "wide": dict(n=150, size=(300, 900, 20, 80)),
    "ties": dict(n=60, size=(3, 40, 2, 40), repeat=40),
    "fans": dict(n=600, size=(5, 80, 5, 80), cross=0.4),
}


@pytest.mark.parametrize("tw", [8, 16, 32, 64])
@pytest.mark.parametrize("shape", sorted(SHAPES))
def test_items_match_oracle(shape, tw):
    w, h = 700, 203
    kw = dict(SHAPES[shape])
    n, size = kw.pop("n"), kw.pop("size")
    for kind, ctx in ((rf.GOURAUD, rf.Context(face_cull=rf.CULL_NONE)),
                      (rf.TEX_GOURAUD, rf.Context(face_cull=rf.CULL_NONE)),
                      (rf.TEXTURED, rf.Context(face_cull=rf.CULL_NONE, depth_test=rf.DEPTH_NONE))):
        d = [tris(len(shape) + tw, n, w, h, size, kind, **kw)]
        vp = mat.viewport(0, 0, w, h)
        assert_parity(gpu_render(d, vp, w, h, ctx=ctx, tile=(tw, 4)), oracle_render(d, vp, w, h, ctx=ctx),
                      what="%s kind %d width %d" % (shape, kind, tw))


def test_lists_that_do_not_fit():
    """More (triangle, tile) pairs than the lists first hold (2^20): the
    masks are walked, then the lists have grown; same image both times."""
    w, h = 1024, 512
    d = [tris(5, 700, w, h, (1500, 2500, 800, 1500))]
    vp = mat.viewport(0, 0, w, h)
    ctx = rf.Context(face_cull=rf.CULL_NONE)
    ref = oracle_render(d, vp, w, h, ctx=ctx)
    dev = rf.Device()
    try:
        # (and the masks that frame left marked do not reach the next one)
        small = [tris(6, 300, 333, 77, (2, 40, 2, 40))]
        vs = mat.viewport(0, 0, 333, 77)
        for _ in range(2):
            assert_parity(gpu_render(d, vp, w, h, ctx=ctx, tile=(8, 4), device=dev), ref)
            assert_parity(gpu_render(small, vs, 333, 77, tile=(32, 4), device=dev),
                          oracle_render(small, vs, 333, 77))
    finally:
        dev.close()


def test_every_raster_group_in_one_batch():
    """Jobs of every shader kind, and of mixed kinds, under the default
    context and another, in an order that interleaves the groups."""
    dev = rf.Device()
    w, h = 150, 90
    vp = mat.viewport(0, 0, w, h)
    jobs, keep = [], []
    try:
        for i in range(18):
            kinds = [i % 6] if i % 6 < 5 else [rf.FLAT, rf.TEX_GOURAUD, rf.GOURAUD]
            ctx = rf.Context(face_cull=rf.CULL_NONE, depth_test=(rf.DEPTH_LESS, rf.DEPTH_GREATER)[i // 6 % 2],
                             depth_clear=float("inf") if i // 6 % 2 == 0 else 0.1)
            ds = [tris(100 + i + k, 80, w, h, (2, 60, 2, 60), k) for k in kinds]
            tg = rf.Framebuf(w, h, device=dev)
            tg.clear(ctx.color_clear, ctx.depth_clear)
            items = []
            for d in ds:
                m = rf.Mesh(d.verts, d.faces, pos_dim=4, device=dev)
                t = rf.Texture(d.tex, device=dev) if d.tex is not None else None
                keep += [m] + ([t] if t else [])
                items.append((m, rf.Shader(d.shader, d.flat_rgba, t), None))
            keep.append(tg)
            jobs.append((rf.Scene(tg, items, vp, ctx), ds, ctx, 1 if rf.GOURAUD_SRGB in kinds else 0))
        stats = rf.render_batch([j[0] for j in jobs], device=dev)
        for (sc, ds, ctx, tol), st in zip(jobs, stats):
            col, dep = sc.target.read()
            assert_parity((col, dep, st), oracle_render(ds, vp, w, h, ctx=ctx), color_tol=tol)
    finally:
        for x in keep:
            x.close()
        dev.close()


@pytest.mark.parametrize("ndraws", [31, 33, 1025, 1100])
def test_many_small_draws(ndraws):
    """Draws of one triangle (a warp's triangles belong to 32 draws), of none
    and of many among them: the lookups of a triangle's and a vertex's draw."""
    rng = np.random.default_rng(ndraws)
    w, h = 256, 160
    draws = []
    for i in range(ndraws):
        n = int(rng.choice([0, 1, 1, 1, 1, 2, 40], p=[.1, .2, .2, .2, .1, .1, .1]))
        d = tris(1000 * ndraws + i, max(n, 1), w, h, (2, 30, 1, 20))
        draws.append(DrawSpec(d.verts, d.faces[:n], rf.GOURAUD, pos_dim=4))
    vp = mat.viewport(0, 0, w, h)
    assert_parity(gpu_render(draws, vp, w, h), oracle_render(draws, vp, w, h), what="%d draws" % ndraws)


@pytest.mark.parametrize("size", [(1, 200, 0.02, 0.6), (0.02, 0.6, 1, 40)])
def test_triangles_between_rows_or_columns(size):
    """Triangles that meet no row (or no column), some of them pieces of
    clipped ones, some past the target's last row."""
    w, h = 300, 120
    d = tris(77, 4000, w, h + 40, size, cross=0.2)
    d.verts[:, 1] *= (h + 40) / h
    vp = mat.viewport(0, 0, w, h)
    for cull in (rf.CULL_BACK, rf.CULL_NONE):
        ctx = rf.Context(face_cull=cull)
        g, o = gpu_render([d], vp, w, h, ctx=ctx), oracle_render([d], vp, w, h, ctx=ctx)
        for depth in (g[1], o[1]):  # (a sliver's 0 / 0: which NaN it is depends on the processor)
            depth[np.isnan(depth)] = np.nan
        assert_parity(g, o, what="cull %d" % cull)


@pytest.mark.parametrize("tile", [(8, 4), (16, 4), (32, 4), (64, 2)])
@pytest.mark.parametrize("kind", [rf.FLAT, rf.GOURAUD, rf.GOURAUD_SRGB])
def test_slanted_tall_triangles(tile, kind):
    """Triangles of 32, 33 and more rows, thin and slanted either way (most of
    their rows miss a tile they are binned into), vertical, and wider than the
    target; on a target smaller than the viewport too."""
    rng = np.random.default_rng(31)
    w, h, n = 400, 300, 500
    dy = rng.choice([31.5, 32.0, 33.0, 34.0, 90.0, 280.0], n)
    dx = rng.choice([0.0, 3.0, -3.0, 40.0, -40.0, 300.0, -300.0, 2000.0, -2000.0], n)
    x, y = rng.uniform(-50, w, n), rng.uniform(-20, h - 20, n)
    px = np.stack([np.stack([x, y], 1), np.stack([x + dx, y + dy], 1),
                   np.stack([x + dx * rng.uniform(0, 1, n) + rng.choice([0.4, 3.0, 30.0], n),
                             y + dy * rng.uniform(0, 1, n)], 1)], 1)
    wv = rng.uniform(1.0, 3.0, (n, 3))
    clip = np.stack([(px[..., 0] / (w / 2.0) - 1.0) * wv, (px[..., 1] / (h / 2.0) - 1.0) * wv,
                     rng.uniform(-0.9, 0.9, (n, 3)) * wv, wv], -1)
    v = np.concatenate([clip, rng.uniform(0, 1, (n, 3, NATTR[kind]))], -1).reshape(3 * n, -1).astype(np.float32)
    d = DrawSpec(v, np.arange(3 * n, dtype=np.uint32).reshape(n, 3), kind, pos_dim=4, flat_rgba=0xFF336699)
    for ctx, tw, th in ((rf.Context(face_cull=rf.CULL_NONE), w, h),
                        (rf.Context(face_cull=rf.CULL_NONE, depth_test=rf.DEPTH_NONE), w - 90, h - 70)):
        vp = mat.viewport(0, 0, w, h)
        g, o = gpu_render([d], vp, tw, th, ctx=ctx, tile=tile), oracle_render([d], vp, tw, th, ctx=ctx)
        for depth in (g[1], o[1]):
            depth[np.isnan(depth)] = np.nan
        assert_parity(g, o, color_tol=1 if kind == rf.GOURAUD_SRGB else 0, what="tile %r" % (tile,))


@pytest.mark.parametrize("n", [1, 2, 3, 9, 40, 300])
def test_few_tall_triangles(n):
    """Few triangles of up to a target's height, several warps to each one's
    rows: chunks of 32 rows, the last one short; clipped pieces among them."""
    w, h = 200, 700
    d = tris(500 + n, n, w, h, (20, 150, 30, 1500), cross=0.2)
    vp = mat.viewport(0, 0, w, h)
    for tile in ((8, 4), (32, 4)):
        g, o = gpu_render([d], vp, w, h, tile=tile), oracle_render([d], vp, w, h)
        assert_parity(g, o, what="%d triangles, tile %r" % (n, tile))


@pytest.mark.parametrize("tw", [8, 16, 32, 64])
@pytest.mark.parametrize("kind", [rf.GOURAUD, rf.TEX_GOURAUD, rf.FLAT])
def test_tables_that_no_row_takes(tw, kind):
    """Whole tables of 32 triangles (and a last, shorter one) that lie in rows
    already covered by nearer ones, in tiles with other rows still clear: no
    round is drawn for them, between tables that are drawn and at the end of a
    tile."""
    w, h, rng = 256, 96, np.random.default_rng(tw)

    def rects(n, y0, y1, wv):  # n triangles across the target, rows y0 .. y1 of every 32 covered
        out = []
        for i in range(n):
            b = 32 * (i % 3)
            out.append([[-300, b + y0], [900, b + y0], [-300, b + 2 * y1 - y0]] if i % 2 else
                       [[900, b + y1], [-300, b + y1], [900, b + 2 * y0 - y1]])
        return np.array(out, np.float64), np.full((n, 3), wv)

    parts = [rects(96, 2, 20, 1.0), rects(32, 21, 31, 1.5)]
    for m in (31, 32, 33, 64, 77):  # farther away, inside the covered rows
        n = 3 * m
        c = np.stack([rng.uniform(0, w, n), 32 * (np.arange(n) % 3) + 11.0], 1)
        px = c[:, None, :] + np.stack([rng.uniform(-90, 90, (n, 3)), np.tile([-6.5, 6.0, 1.0], (n, 1))], -1)
        parts.append((px, rng.uniform(2.0, 3.0, (n, 3))))
        parts.append(rects(3, 24, 30, 1.4 - 0.01 * m / 31))
    parts.append(parts[4])
    px, wv = (np.concatenate(x) for x in zip(*parts))
    n = len(px)
    clip = np.stack([(px[..., 0] / (w / 2.0) - 1.0) * wv, (px[..., 1] / (h / 2.0) - 1.0) * wv, 0.0 * wv, wv], -1)
    v = np.concatenate([clip, rng.uniform(0, 1, (n, 3, NATTR[kind]))], -1).reshape(3 * n, -1).astype(np.float32)
    tex = scenes.noise_texture(64, 3) if kind == rf.TEX_GOURAUD else None
    d = DrawSpec(v, np.arange(3 * n, dtype=np.uint32).reshape(n, 3), kind, pos_dim=4, flat_rgba=0xFF336699, tex=tex)
    vp, ctx = mat.viewport(0, 0, w, h), rf.Context(face_cull=rf.CULL_NONE)
    o = oracle_render([d], vp, w, h, ctx=ctx)
    assert o[2]["frags_o"] > 0
    for _ in range(3):
        assert_parity(gpu_render([d], vp, w, h, ctx=ctx, tile=(tw, 4)), o, what="width %d" % tw)


@pytest.mark.parametrize("large", [(rf.GOURAUD, rf.TEX_GOURAUD), (rf.FLAT, rf.GOURAUD, rf.TEXTURED, rf.TEX_GOURAUD,
                                                                  rf.GOURAUD_SRGB)])
@pytest.mark.parametrize("graphs", [False, True])
def test_large_and_small_groups_in_one_batch(graphs, large):
    """Raster groups large enough for kernels of their own, of some kinds or of
    every one, in both contexts, and small ones that go together: replayed too."""
    dev = rf.Device()
    dev.set_graphs(graphs)
    w, h = 260, 130
    vp = mat.viewport(0, 0, w, h)
    jobs, keep = [], []
    try:
        kinds = [rf.FLAT, rf.GOURAUD, rf.TEXTURED, rf.TEX_GOURAUD, rf.GOURAUD_SRGB]
        for i, (k, test, n) in enumerate([(k, t, n) for n in (60, 33000, 90) for t in (rf.DEPTH_LESS, rf.DEPTH_GREATER)
                                          for k in kinds if n == 60 or k in large]):
            ctx = rf.Context(face_cull=rf.CULL_NONE, depth_test=test,
                             depth_clear=float("inf") if test == rf.DEPTH_LESS else 0.1)
            d = tris(300 + i, n, w, h, (1, 6, 1, 6) if n > 1000 else (2, 60, 2, 60), k)
            tg = rf.Framebuf(w, h, device=dev)
            m = rf.Mesh(d.verts, d.faces, pos_dim=4, device=dev)
            t = rf.Texture(d.tex, device=dev) if d.tex is not None else None
            keep += [tg, m] + ([t] if t else [])
            jobs.append((rf.Scene(tg, [(m, rf.Shader(d.shader, d.flat_rgba, t), None)], vp, ctx),
                         oracle_render([d], vp, w, h, ctx=ctx), ctx, 1 if k == rf.GOURAUD_SRGB else 0))
        for _ in range(3):
            for sc, _, ctx, _ in jobs:
                sc.target.clear(ctx.color_clear, ctx.depth_clear)
            stats = rf.render_batch([j[0] for j in jobs], device=dev)
            for (sc, ref, ctx, tol), st in zip(jobs, stats):
                col, dep = sc.target.read()
                assert_parity((col, dep, st), ref, color_tol=tol)
    finally:
        for x in keep:
            x.close()
        dev.close()


@pytest.mark.parametrize("tw", [8, 32])
@pytest.mark.parametrize("kind", sorted(NATTR))
def test_triangles_past_the_top(kind, tw):
    """Triangles whose first rows lie above the target (all of them drawn in row
    0, one lane's): of one such row and of hundreds, the two halves' both, in
    both contexts."""
    w, h = 210, 70
    parts = [tris(60 + i, 60, w, 2 * h, (4, 80, y0, y1), kind) for i, (y0, y1) in enumerate(((1, 6), (20, 90), (200, 700)))]
    v = np.concatenate([p.verts for p in parts])
    d = DrawSpec(v, np.arange(len(v), dtype=np.uint32).reshape(-1, 3), kind, pos_dim=4, flat_rgba=0xFF336699,
                 tex=parts[0].tex)
    vp = mat.viewport(0, -h, w, h)
    for ctx in (rf.Context(face_cull=rf.CULL_NONE), rf.Context(face_cull=rf.CULL_NONE, depth_test=rf.DEPTH_NONE)):
        g, o = gpu_render([d], vp, w, h, ctx=ctx, tile=(tw, 4)), oracle_render([d], vp, w, h, ctx=ctx)
        assert_parity(g, o, color_tol=1 if kind == rf.GOURAUD_SRGB else 0, what="kind %d" % kind)
