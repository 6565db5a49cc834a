"""The tile masks from frame to frame on one device, against the oracle bit for
bit: they are zeroed when they are allocated, and by the list pass after that."""
import numpy as np
import pytest

import retrofire_gb300 as rf
from retrofire_gb300 import mat
from rfhelp import DrawSpec, assert_parity, gpu_render, oracle_render

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    from retrofire_gb300 import build
    build.build()
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")


def boxes(seed, n, w, h, size):
    """n Gouraud triangles of about size px at random places of a w x h target."""
    rng = np.random.default_rng(seed)
    px = rng.uniform([0, 0], [w, h], (n, 2))[:, None, :] + rng.uniform(-0.5, 0.5, (n, 3, 2)) * size
    wv = rng.uniform(1.0, 3.0, (n, 3))
    clip = np.stack([(px[..., 0] / (w / 2.0) - 1.0) * wv, (px[..., 1] / (h / 2.0) - 1.0) * wv,
                     rng.uniform(-0.9, 0.9, (n, 3)) * wv, wv], -1)
    v = np.concatenate([clip, rng.uniform(0, 1, (n, 3, 3))], -1).reshape(3 * n, 7).astype(np.float32)
    return DrawSpec(v, np.arange(3 * n, dtype=np.uint32).reshape(n, 3), rf.GOURAUD, pos_dim=4)


@pytest.mark.parametrize("sort", [rf.SORT_NONE, rf.SORT_BACK_TO_FRONT])
def test_masks_that_grow(sort):
    """Step by step larger masks, a small frame after each step."""
    dev = rf.Device()
    ctx = rf.Context(face_cull=rf.CULL_NONE, depth_sort=sort,
                     depth_test=rf.DEPTH_NONE if sort else rf.DEPTH_LESS)
    small, vs = boxes(1, 50, 100, 70, 20), mat.viewport(0, 0, 100, 70)
    ref = oracle_render([small], vs, 100, 70, ctx=ctx)
    try:
        for i, (n, w, h) in enumerate(((300, 200, 120), (1100, 333, 257), (5000, 640, 360), (20000, 800, 600))):
            d, vp = boxes(2 + i, n, w, h, 12), mat.viewport(0, 0, w, h)
            g = gpu_render([d], vp, w, h, ctx=ctx, tile=(16, 4), device=dev)
            assert_parity(g, oracle_render([d], vp, w, h, ctx=ctx), what="%d triangles" % n)
            assert_parity(gpu_render([small], vs, 100, 70, ctx=ctx, tile=(8, 4), device=dev), ref,
                          what="50 after %d" % n)
    finally:
        dev.close()


@pytest.mark.parametrize("sort", [rf.SORT_NONE, rf.SORT_BACK_TO_FRONT])
def test_lists_past_their_room(sort):
    """More (triangle, tile) pairs than the triangle lists first hold: the
    rasteriser walks the masks, which stay marked; the next frame, smaller or
    larger, starts from zero, and the same frame again fits its grown lists."""
    w, h, n = 1024, 512, 700
    tiles = (w // 8) * (h // 32)
    rng = np.random.default_rng(9)
    # Triangles (0, 0), (2900, 0), (0, 1450) of a 3000 x 1500 viewport, corners
    # moved outwards by up to 40 px, every other one turned: all cover the target.
    vw, vh = 3000.0, 1500.0
    px = np.array([[1.0, 1.0], [2900.0, 1.0], [1.0, 1450.0]]) + rng.uniform([-0.9, -0.9], [40, 40], (n, 3, 2)) * \
        np.array([[0, 0], [1, 0], [0, 1]])
    px[:, 0] -= rng.uniform(0, 0.9, (n, 2))
    for a, b in ((0, 1), (1, 2), (2, 0)):  # the target's corners lie inside every edge
        for c in ((1, 1), (w, 1), (1, h), (w, h)):
            e, f = px[:, b] - px[:, a], np.array(c, float) - px[:, a]
            assert (e[:, 0] * f[:, 1] - e[:, 1] * f[:, 0] >= -1e-6).all()
    assert n * tiles > max(4 * n, 1 << 20)  # the room of a new context
    px[::2] = px[::2, ::-1]
    wv = rng.uniform(1.0, 3.0, (n, 1)).repeat(3, 1) * rng.uniform(0.95, 1.05, (n, 3))
    clip = np.stack([(px[..., 0] / (vw / 2) - 1.0) * wv, (px[..., 1] / (vh / 2) - 1.0) * wv,
                     rng.uniform(-0.9, 0.9, (n, 3)) * wv, wv], -1)
    v = np.concatenate([clip, rng.uniform(0, 1, (n, 3, 3))], -1).reshape(3 * n, 7).astype(np.float32)
    big = DrawSpec(v, np.arange(3 * n, dtype=np.uint32).reshape(n, 3), rf.GOURAUD, pos_dim=4)
    ctx = rf.Context(face_cull=rf.CULL_NONE, depth_sort=sort,
                     depth_test=rf.DEPTH_NONE if sort else rf.DEPTH_LESS)
    vp = mat.viewport(0, 0, int(vw), int(vh))
    ref = oracle_render([big], vp, w, h, ctx=ctx)
    for after in ((300, 333, 77, (32, 4)), (20000, 1280, 720, (16, 4))):
        d, va = boxes(4, after[0], after[1], after[2], 15), mat.viewport(0, 0, after[1], after[2])
        oa = oracle_render([d], va, after[1], after[2], ctx=ctx)
        dev = rf.Device()
        try:
            for what in ("walked", "grown"):
                assert_parity(gpu_render([big], vp, w, h, ctx=ctx, tile=(8, 4), device=dev), ref, what=what)
                assert_parity(gpu_render([d], va, after[1], after[2], ctx=ctx, tile=after[3], device=dev), oa,
                              what="after " + what)
        finally:
            dev.close()
