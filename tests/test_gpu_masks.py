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
