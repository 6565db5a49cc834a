"""CPU test of a rule of the frame's launches (rf_kernels.cuh, launch_next): a
kernel that comes up while the one before it drains reads what that one writes
by plain loads.  Loads the compiler may take for read-only (__ldg, parameters
that are __restrict__ and not written) need memory that nobody writes while the
kernel is resident."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "retrofire_gb300", "csrc")

# file, kernel, what it reads of the kernel launched before it
FRESH = [
    ("rf_kernels.cu", "k_vertex", ["draws"]),  # k_cull
    ("rf_kernels.cu", "k_clip", ["coc"]),  # k_vertex
    ("rf_kernels.cu", "k_clip_poly", ["queue"]),  # k_clip
    ("rf_kernels.cu", "k_scan_blocks", ["in"]),  # k_clip_poly, k_rs_hist
    ("rf_kernels.cu", "k_scan_add", ["sums"]),  # k_scan_sums
    ("rf_kernels.cu", "k_setup", ["tcnt", "toff", "tpoly", "pool", "perm", "ptri"]),  # k_clip_poly, the sort
    ("rf_kernels.cu", "k_bin_small", ["prims", "live_small", "small_n"]),  # k_setup
    ("rf_kernels.cu", "k_bin", ["live", "live_n", "prims"]),  # k_setup, k_bin_small
    ("rf_kernels.cu", "k_tile_lists", ["ent", "marks"]),  # k_bin
    ("rf_kernels.cu", "k_stats_fold", ["js"]),  # k_raster
    ("rf_sort.cu", "k_draw_counts", ["toff", "counters"]),  # the scan
    ("rf_sort.cu", "k_rs_hist", ["keys"]),  # k_dsort_keys, k_rs_scatter
    ("rf_sort.cu", "k_rs_scatter", ["kin", "vin", "cnt"]),  # k_dsort_keys, k_rs_scatter, the scan
    ("rf_lines.cu", "k_line_setup", ["cpos", "coc"]),  # k_vertex
    ("rf_lines.cu", "k_line_raster", ["recs", "mask"]),  # k_line_setup
]


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def kernel(text, name):
    """A kernel's parameters and body."""
    m = re.search(r"__global__[^;{]*?\b%s\(([^{]*?)\)\s*\{" % name, text, re.S)
    assert m, name
    end, depth = m.end(), 1
    while depth:
        depth += {"{": 1, "}": -1}.get(text[end], 0)
        end += 1
    return m.group(1), text[m.end():end]


@pytest.mark.parametrize("name,kern,params", FRESH, ids=[k for _, k, _ in FRESH])
def test_predecessors_data_by_plain_loads(name, kern, params):
    sig, body = kernel(source(name), kern)
    decls = {d.split()[-1].lstrip("*"): d for d in sig.replace("\n", " ").split(",")}
    for p in params:
        assert "__restrict__" not in decls[p], decls[p]
        assert not re.search(r"__ld(g|cs|cg|lu|cv|ca)\(\s*\(?%s\b" % p, body), p


def test_raster_reads_the_lists_by_plain_loads():
    """k_raster's arguments come in a struct; k_tile_lists writes list, segs,
    items, first and nfirst."""
    text = source("rf_raster.cuh")
    for m in re.finditer(r"__ldg\(([^;]*)", text):
        assert not re.search(r"\b(list|segs|seg|items|first|nfirst|ent)\b", m.group(1)), m.group(0)


def test_every_kernel_launched_early_waits_first():
    for name in ("rf_kernels.cu", "rf_sort.cu", "rf_lines.cu"):
        text = source(name)
        for kern in set(re.findall(r"RF_NEXT\((k_\w+)", text)) | {k for f, k, _ in FRESH if f == name}:
            _, body = kernel(text, kern)
            assert re.match(r"\s*(using namespace \w+;\s*)?(rfd::)?grid_begin\(\);", body), kern
