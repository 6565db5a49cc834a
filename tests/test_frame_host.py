"""CPU tests of the frame code (retrofire_gb300/csrc/rf_api.cu) against a CUDA
runtime of host memory (tests/csrc/frame_shim.cpp): what its buffers hold from
frame to frame."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    inc = os.path.join(os.path.dirname(os.path.dirname(NVCC)), "include")
    if not os.path.exists(os.path.join(inc, "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    out = str(tmp_path_factory.mktemp("shim") / "libframe.so")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-Wl,-Bsymbolic",
                           "-I" + inc, os.path.join(HERE, "csrc", "frame_shim.cpp"), "-o", out])
    L = C.CDLL(out)
    L.shim_frames.argtypes = [C.c_void_p, C.c_uint32, C.POINTER(C.c_uint64)]
    L.shim_frames.restype = C.c_uint32
    L.shim_zero_blocks.argtypes = [C.c_uint64, C.c_int, C.c_uint32, C.c_int]
    L.shim_zero_blocks.restype = C.c_uint32
    L.shim_draws.argtypes = [C.c_void_p, C.c_uint32, C.c_uint64, C.POINTER(C.c_uint64)]
    L.shim_alloc_fails.argtypes = [C.c_uint32, C.POINTER(C.c_uint64)]
    L.shim_event_fails.argtypes = [C.c_uint32, C.POINTER(C.c_int32)]
    L.shim_groups.argtypes = [C.c_void_p, C.c_uint32, C.c_void_p, C.POINTER(C.c_uint32), C.POINTER(C.c_uint64)]
    L.shim_trials.argtypes = [C.c_uint32, C.c_int, C.c_int32, C.c_char_p, C.c_uint32]
    L.shim_pick.argtypes = [C.c_void_p, C.c_int]
    L.shim_refused.argtypes = [C.c_uint32, C.c_uint32, C.POINTER(C.c_uint64)]
    return L


def frames(L, rows):
    """(mask words found set, setup passes, masks grown in place) of a run of
    (ntri, w, h, depth_sort, clipped, fails) frames."""
    a = np.ascontiguousarray(rows, np.uint32)
    out = (C.c_uint64 * 3)()
    assert L.shim_frames(a.ctypes.data, len(a), out) == 0
    return tuple(out)


@pytest.mark.parametrize("sort", [0, 1])
def test_grown_masks_start_zero(shim, sort):
    """Masks that grow, step by step, onto the address they had: every frame
    finds them zero, those after the largest too."""
    rows = [(n, w, h, sort, 1, 0) for n, w, h in
            ((40, 64, 64), (700, 320, 240), (40, 64, 64), (9000, 640, 480), (70000, 640, 480), (40, 64, 64))]
    dirty, setups, grown = frames(shim, rows)
    assert setups == len(rows)
    assert grown >= 2  # (the case this is about)
    assert dirty == 0


def test_masks_grown_by_clipped_pieces(shim):
    """A depth-sorted frame's masks grow a second time, by its clipped
    triangles, in the middle of the frame."""
    dirty, setups, grown = frames(shim, [(3000, 320, 240, 1, 1, 0), (3000, 320, 240, 1, 7, 0), (3000, 320, 240, 0, 1, 0)])
    assert (dirty, setups) == (0, 3) and grown >= 1


@pytest.mark.parametrize("sort", [0, 1])
def test_frame_cut_short(shim, sort):
    """A frame that fails between marking and reading the masks: the next
    one finds them zero, larger or smaller."""
    for after in (40, 700, 9000):
        dirty, setups, _ = frames(shim, [(700, 320, 240, sort, 1, 0), (700, 320, 240, sort, 1, 1), (after, 320, 240, 0, 1, 0)])
        assert (dirty, setups) == (0, 3)


def test_new_masks_not_zeroed(shim):
    """A frame that fails between allocating larger masks and zeroing them:
    the next one zeroes them, though they are large enough by then."""
    dirty, setups, _ = frames(shim, [(40, 64, 64, 0, 1, 0), (9000, 640, 480, 0, 1, 2), (9000, 640, 480, 0, 1, 0)])
    assert (dirty, setups) == (0, 2)


@pytest.mark.parametrize("mask_mb", [0, 1, 16, 300, 4000])
@pytest.mark.parametrize("ntiles", [1, 60, 4080, 1 << 20])
def test_zeroing_grid_covers_masks_left_marked(shim, mask_mb, ntiles):
    """A frame's zeroing launch after one that left the masks marked: the whole
    chip clears large masks, whatever target the frame is for; small masks and
    few tiles take few blocks."""
    nsm, n16 = 152, mask_mb << 16
    b = shim.shim_zero_blocks(n16, 0, ntiles, nsm)
    assert b >= min(n16 // 256, nsm) and b * 256 >= min(ntiles, nsm * 8 * 256)
    assert b <= max(2 * nsm, min(ntiles // 256 + 2, 8 * nsm)) and b <= (n16 + ntiles) // 256 + 2


COUNTS = [1, 40, 101, 300, 5000, 7, 20000, 5000, 20, 300]


@pytest.mark.parametrize("limit", [1 << 40, 4096, 1 << 20])
def test_descriptors_arrive(shim, limit):
    """Every draw's descriptor reaches the device as it was built, whatever the
    frames before needed, and whether or not memory can be page-locked."""
    a, out = np.array(COUNTS, np.uint32), (C.c_uint64 * 3)()
    assert shim.shim_draws(a.ctypes.data, len(a), limit, out) == 0
    assert (out[0], out[1]) == (0, sum(COUNTS))


@pytest.mark.parametrize("good", [0, 1, 255, 256, 257, 3000])
def test_refused_calls_lock_no_memory_for_what_they_claim(shim, good):
    """A call whose count is wrong ends at its first bad draw with that draw's
    status, and page-locks memory for the draws before it at most."""
    n = C.c_uint64()
    assert shim.shim_refused(good, 0xFFFFFFFF, C.byref(n)) == 1  # RF_ERR_BAD_HANDLE
    assert n.value <= 65536 + 2 * 16 * 1.25 * 200 * good


@pytest.mark.parametrize("k", range(40))
def test_frame_after_one_out_of_memory(shim, k):
    """A first frame whose k-th allocation fails, then one that gets its memory:
    it has counters, and they are zero."""
    out = (C.c_uint64 * 3)()
    st = shim.shim_alloc_fails(k, out)
    assert st in (0, 4)  # RF_ERR_OOM; 0: the frame makes fewer
    assert tuple(out) == (0, 0, 0)


@pytest.mark.parametrize("k", range(6))
def test_frame_after_one_short_of_events(shim, k):
    """A first batch of two raster groups whose k-th event cannot be made, then
    one that gets its events: it is rendered."""
    out = C.c_int32()
    st = shim.shim_event_fails(k, C.byref(out))
    assert (st, out.value) in ((4, 0), (0, 0))  # RF_ERR_OOM; 0: the batch makes fewer


FLAT, GOURAUD, SRGB, MIXED = 0, 1, 4, 5


@pytest.mark.parametrize("jobs,groups", [  # (shader, default context, triangles)
    ([(GOURAUD, 1, 100)], [(GOURAUD, 1, 100)]),
    ([(FLAT, 1, 100), (GOURAUD, 1, 200)], [(MIXED, 1, 300)]),
    ([(FLAT, 1, 5), (GOURAUD, 0, 7)], [(FLAT, 1, 5), (GOURAUD, 0, 7)]),
    ([(k, c, 10) for k in (SRGB, FLAT, GOURAUD) for c in (0, 1)], [(MIXED, 1, 30), (MIXED, 0, 30)]),
    ([(GOURAUD, 0, 40), (GOURAUD, 1, 40)], [(GOURAUD, 1, 40), (GOURAUD, 0, 40)]),
    ([(FLAT, 1, 33000), (GOURAUD, 1, 10), (GOURAUD, 1, 20)], [(FLAT, 1, 33000), (GOURAUD, 1, 30)]),
    ([(FLAT, 1, 9), (GOURAUD, 1, 20000), (GOURAUD, 1, 20000), (SRGB, 1, 9)], [(GOURAUD, 1, 40000), (MIXED, 1, 18)]),
])
def test_raster_groups(shim, jobs, groups):
    """Groups of few triangles are one of mixed kinds, the others a group each,
    on a stream each; the groups of one kind share their setup launches."""
    a, out = np.array(jobs, np.uint32), np.zeros(64, np.uint32)
    streams, k = C.c_uint32(), C.c_uint64()
    n = shim.shim_groups(a.ctypes.data, len(a), out.ctypes.data, C.byref(streams), C.byref(k))
    assert [tuple(r) for r in out[:3 * n].reshape(n, 3).tolist()] == groups
    assert streams.value == n
    kinds = len({g[0] for g in groups})
    # a mesh's box two, zero, vertex, clip two, lists, the stats, three a kind, one a group
    assert k.value == 2 * len(jobs) + 6 + 3 * kinds + n


@pytest.mark.parametrize("graphs,sort,timed", [(0, 0, "ERE"), (1, 0, "EGE"), (0, 1, "ERE"), (1, 1, "ERE")])
def test_trials_time_the_frame_alone(shim, graphs, sort, timed):
    """The frames that pick a tile width: loading its kernels, capturing,
    instantiating and uploading its graph all come before the first event."""
    log = C.create_string_buffer(4096)
    assert shim.shim_trials(9, graphs, sort, log, len(log)) == 0
    f = log.value.decode().split("|")
    for trial in f[1:5]:
        assert trial.count("E") == 2 and trial[trial.index("E"):] == timed, f
        assert "L" in trial[:trial.index("E")]
    assert not any("E" in x or "L" in x for x in f[:1] + f[5:])


@pytest.mark.parametrize("us,replayed,launched", [
    ((100, 100, 100, 100), 8, 8), ((100, 98, 96, 110), 32, 8), ((59.5, 54.8, 62.2, 70), 16, 8), ((140, 120, 118, 150), 16, 16),
    ((1000, 975, 960, 970), 32, 32), ((100, 90, 80, 68), 64, 64), ((100, 200, 300, 400), 8, 8)])
def test_a_wider_tile_has_to_be_clearly_faster(shim, us, replayed, launched):
    a = np.array(us, np.float32) / 1000
    assert (shim.shim_pick(a.ctypes.data, 1), shim.shim_pick(a.ctypes.data, 0)) == (replayed, launched)
