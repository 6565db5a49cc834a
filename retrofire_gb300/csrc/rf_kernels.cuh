// rf_kernels.cuh — constants and launch helpers shared by rf_kernels.cu and
// the C-ABI driver rf_api.cu.
#ifndef RF_KERNELS_CUH
#define RF_KERNELS_CUH

#include <cuda_runtime.h>
#include <stdint.h>

#include "rf_internal.cuh"

// Mirrors of the public enums in include/rfgpu.h.
#define RF_K_FLAT 0
#define RF_K_GOURAUD 1
#define RF_K_TEXTURED 2
#define RF_K_TEX_GOURAUD 3
#define RF_K_GOURAUD_SRGB 4
#define RF_K_ANY 5  // rasteriser kernel that dispatches on each triangle's kind
#define RF_K_REPEAT_POT 0
#define RF_K_CLAMP 1
#define RF_K_ONCE 2
#define RF_K_ARGB8888 0
#define RF_K_XRGB8888 1
#define RF_K_RGBA8888 2
#define RF_K_BGRA8888 3
#define RF_K_DEPTH_NONE 0
#define RF_K_DEPTH_LESS 1
#define RF_K_DEPTH_EQUAL 2
#define RF_K_DEPTH_GREATER 3
#define RF_K_CULL_NONE 0
#define RF_K_CULL_BACK 1
#define RF_K_CULL_FRONT 2
#define RF_K_DRAW_CULL_BBOX 1u

#define RF_NO_POLY 0xFFFFFFFFu
// Scanline y origins beyond +-2^22 px are outside the supported domain: the
// row arithmetic y0r + j must stay exact in f32.  Such halves count in oob.
#define RF_MAX_COORD 4194304.0f
#define RF_RASTER_MAX_THREADS 256
// The jobs of a frame are laid out by raster group: one shader kind (or
// RF_K_ANY: jobs that mix kinds) and one context (the default one on a depth
// target, or any other).  Every group has a raster launch of its own,
// specialised for both, and its own part of the work list; the groups of one
// kind share setup and binning launches and live lists.
#define RF_MAX_GROUPS (2 * (RF_K_ANY + 1))
struct RasterGroup {
    int32_t kind;
    bool fast;
    uint32_t tile0, ntiles;
    uint32_t block0, nblocks;  // setup blocks
    uint32_t ntri;             // triangles
};

// counters[] slots
#define RF_CNT_POOL 0     // pool slots used
#define RF_CNT_POOLOVF 1  // polygons dropped for lack of pool slots
#define RF_CNT_POLYOVF 2  // polygons that exceeded RF_POLY_CAP vertices
#define RF_CNT_BADIDX 3   // triangles with an out-of-range vertex index
#define RF_CNT_PRIMS 4    // total output prims (scan total)
#define RF_CNT_QUEUE 5    // tile queue head of the line pass
#define RF_CNT_ROWSOVF 6  // triangles rasterised without row records (buffer full)
#define RF_CNT_MASKDIRTY 9 // nonzero: the tile masks were not left zero
#define RF_CNT_CLIPQ 10   // triangles queued for clipping
#define RF_CNT_QUEUE_G 16     // + g: work-list queue head of raster group g
#define RF_CNT_ITEMS_G (RF_CNT_QUEUE_G + RF_MAX_GROUPS)  // + g: its heavy tiles and crowded tiles' slices
#define RF_CNT_LIVE_G (RF_CNT_ITEMS_G + RF_MAX_GROUPS)   // + g, a kind's first group: live triangles, binned a warp each
#define RF_CNT_LIVE_MID_G (RF_CNT_LIVE_G + RF_MAX_GROUPS)  // + g: ... sixteen lanes each (at most 16 rows)
#define RF_CNT_N (RF_CNT_LIVE_MID_G + RF_MAX_GROUPS)
#define RF_SCAN_BLOCK_ITEMS 4096u  // values one scan block takes (one launch instead of three)

namespace rfk {
#if defined(__CUDACC__)
// A launch that may start while the kernel before it on the stream drains
// (programmatic dependent launch): its blocks come up and wait in
// grid_begin() (rf_device.cuh) until that kernel has finished, so the launch
// latency and the wait for the last block do not add up.  Every kernel
// launched here calls grid_begin() first.  It is resident while the kernel
// before it still writes, so it reads what that one writes by plain loads: not
// through __ldg, nor from a parameter that is const and __restrict__ (or only
// read, and __restrict__), whose memory must not change while the kernel lives.
// What earlier kernels wrote is complete by then: each lets its successor come
// up only after its own wait.
template <class... P, class... A>
cudaError_t launch_next(void (*k)(P...), uint32_t blocks, uint32_t threads, size_t smem, cudaStream_t s, A... a) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(blocks);
    c.blockDim = dim3(threads);
    c.dynamicSmemBytes = smem;
    c.stream = s;
    c.attrs = &at;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, k, static_cast<P>(a)...);
}
#define RF_NEXT(...)                                          \
    do {                                                      \
        const cudaError_t next_ = rfk::launch_next(__VA_ARGS__); \
        if (next_ != cudaSuccess) return next_;               \
    } while (0)
#endif
// Zeroes what a frame accumulates into: the jobs' stats slots js[0 .. njobs),
// the tiles' entry counts, totals[0..2) (row words, list entries), *marks
// (the binning pass's total of (triangle, tile) bits), the frame's counters
// and -- when the last frame left them dirty, or with `masks` -- the whole mask
// buffer (mask_words, a multiple of 4).  launch_vertex clears the dirty mark
// (counters: nullptr for none).
// Blocks of 256: for the tiles' counts, and for the masks' n16 16-byte words, up to
// eight blocks a multiprocessor where they are certain to be cleared and two
// where only the device knows (a block with nothing to clear ends after one
// load).
inline uint32_t zero_blocks(size_t n16, bool masks, uint32_t ntiles, int nsm) {
    auto upto = [&](size_t work, int per_sm) {
        const size_t b = (work + 255) / 256 + 1, most = (size_t)nsm * per_sm;
        return b < most ? b : most;
    };
    const size_t a = upto(ntiles, 8), b = upto(n16, masks ? 8 : 2);
    return (uint32_t)(a > b ? a : b);
}
cudaError_t launch_zero(uint32_t *mask, size_t mask_words, bool masks, StatsDev *js, uint32_t njobs,
                        unsigned long long *tacc, uint32_t ntiles, unsigned long long *totals,
                        unsigned long long *marks, uint32_t *counters, int nsm, cudaStream_t s);
cudaError_t launch_vertex(const DrawDev *draws, uint32_t nd, uint32_t nv, float4 *cpos,
                          uint8_t *coc, uint32_t *counters, int nsm, cudaStream_t s);
// Clip status, the clipping of the triangles that cross a plane, and each
// input triangle's fan count tcnt.  queue: room for nt triangle indices.
// place: each input triangle's first output slot into toff, taken from a
// running total (counters[RF_CNT_PRIMS]): one slot for a visible triangle,
// RF_MAX_FAN for one that is clipped (its fan fills the first tcnt), the
// triangles' blocks in any order -- every later pass finds a triangle's
// outputs through toff and tcnt.  Otherwise toff is left to the scan
// (launch_scan), which packs the outputs in clipped order for the depth
// sort, and the queue may be the scan's output array.
cudaError_t launch_clip(const DrawDev *draws, uint32_t nd, uint32_t nt, const float4 *cpos,
                        const uint8_t *coc, uint32_t *tcnt, uint32_t *tpoly, uint32_t *queue,
                        PolyVert *pool, uint32_t pool_cap, uint32_t *counters, int nsm, cudaStream_t s,
                        uint32_t *toff, bool place);
// BBox::of a mesh's positions (the first three floats of each vertex of
// stride floats) into bbox[0..6); bbox[6 ..) is scratch for the per-block
// parts: bbox holds RF_MESH_BBOX_FLOATS floats.
#define RF_MESH_BBOX_BLOCKS 64u
#define RF_MESH_BBOX_FLOATS (6u + 6u * RF_MESH_BBOX_BLOCKS)
cudaError_t launch_mesh_bbox(const float *verts, uint32_t nverts, uint32_t stride, float *bbox,
                             cudaStream_t s);
size_t scan_scratch_words(uint32_t n);
cudaError_t launch_scan(const uint32_t *in, uint32_t *out, uint32_t n, uint32_t *scratch,
                        uint32_t *total, cudaStream_t s);
// Triangle setup (k_setup: also the row records and tile bits of triangles
// of a few rows), then scanline statistics, row records and tile binning of
// the others (k_bin_small for at most 16 rows, then k_bin), per shader kind.
// rows holds rows_cap words; rows_total receives the words the frame asked
// for, each triangle's records placed by k_setup from it (rows_total[1] is
// the lists' cursor); live (room for twice every output triangle) receives
// the index of each triangle left for the binning pass, kind after kind:
// those for k_bin (counters[RF_CNT_LIVE_G + g]) in its first half, the regular
// ones with at most 16 rows on the target (counters[RF_CNT_LIVE_MID_G + g])
// in its second; *marks receives the (triangle, tile) bits set in all.
// sorted: perm and ptri give the depth-sorted order (rf_sort.cu).
cudaError_t launch_setup(const DrawDev *draws, uint32_t nd, const JobDev *jobs, uint32_t nj,
                         const RasterGroup *groups, uint32_t ng, uint32_t nt, uint32_t tile_w, const float4 *cpos,
                         const uint32_t *tcnt, const uint32_t *toff, const uint32_t *tpoly, const PolyVert *pool,
                         PrimRec *prims, unsigned long long *rows_total, uint32_t *rows,
                         unsigned long long rows_cap, RasterPrim *rprims, uint2 *ent, uint32_t *mask, uint32_t *live,
                         unsigned long long *marks, StatsDev *stats, uint32_t *counters, int nsm,
                         cudaStream_t s, const uint32_t *perm = nullptr, const uint32_t *ptri = nullptr);
// The tiles' triangle lists and the rasteriser's work list, from the tile
// masks and the marks total (slots: the warps the rasteriser keeps resident,
// about).
// Lists: the set bits of every tile's mask as entries, one per input
// triangle, in submission order: ent[t], written by the setup and binning
// passes -- x: its first output triangle | (its outputs - 1) <<
// RF_ENT_SHIFT, y: the depth bound of a single output (RasterPrim::zmax),
// NaN for more.  A tile's list comes in J.nseg pieces (segs[J.seg_base + tile
// * J.nseg + k]: offset, entries), each placed by atomics on *cursor; a piece
// that would end past cap entries is marked RF_SEG_WALK instead and the
// rasteriser walks its masks.  The masks are left zero for the next frame,
// but for the pieces marked: then counters[RF_CNT_MASKDIRTY] is set and
// the next launch_zero clears them all.  tacc (a word pair per tile, zeroed
// by launch_zero) gathers a tile's entries over its pieces.
// Work list: items (room for (RF_SPLIT_K + 1) * ntiles): items[ntiles ..
// ntiles + extra) first -- heavy tiles (tile << RF_ITEM_SHIFT) and the row
// slices of crowded tiles (tile << RF_ITEM_SHIFT | k, k = 1 .. RF_SPLIT_K) --
// then items[0 .. ntiles): tile t << RF_ITEM_SHIFT in index order,
// RF_ITEM_SKIP for the tiles already listed; extra is
// counters[RF_CNT_ITEMS_G + g], the list per raster group g: its tiles are
// tile0 .. tile0 + n and its first part starts at ntiles + RF_SPLIT_K * tile0.
#define RF_ENT_SHIFT 29u
#define RF_ENT_MASK ((1u << RF_ENT_SHIFT) - 1u)
static_assert(RF_MAX_FAN <= 8, "an entry holds a fan's size");
#define RF_SEG_WALK 0xFFFFFFFFu
cudaError_t launch_lists(const JobDev *jobs, uint32_t nj, uint32_t *mask, uint32_t ntiles, uint32_t npieces,
                         const uint2 *ent, unsigned long long *tacc, const unsigned long long *marks, uint32_t slots, uint32_t *items, uint32_t *counters,
                         uint2 *segs, uint2 *list, unsigned long long *cursor, unsigned long long cap,
                         cudaStream_t s);
#ifndef RF_SPLIT_K
#define RF_SPLIT_K 4  // row slices of a crowded tile (RF_TILE_H / RF_SPLIT_K rows each)
#endif
// A work item is tile << RF_ITEM_SHIFT | k (k = 0: the whole tile, 1..RF_SPLIT_K: a slice).
#define RF_ITEM_SHIFT (RF_SPLIT_K < 8 ? 3u : 4u)
static_assert(RF_TILE_H % RF_SPLIT_K == 0 && RF_SPLIT_K < 16, "row slices");
#define RF_ITEM_SKIP 0xFFFFFFFEu  // a work-list entry taken elsewhere in the list
#define RF_MAX_TILES (1u << (31 - RF_ITEM_SHIFT))  // tiles of one frame or batch
// The launchers per tile width (rf_raster.cuh).
#define RF_RASTER_PARAMS                                                                              \
    const JobDev *jobs, uint32_t nj, const DrawDev *draws, const PrimRec *prims, const RasterPrim *rprims, \
        const uint32_t *rows, const uint2 *ent, const uint32_t *mask, const uint2 *segs,                 \
        const uint2 *list, const uint32_t *items, uint32_t ntiles, const uint32_t *first, const uint32_t *nfirst,          \
        uint32_t *queue, StatsDev *stats, uint32_t warps, int nsm, cudaStream_t s
#define RF_RASTER_ARGS \
    jobs, nj, draws, prims, rprims, rows, ent, mask, segs, list, items, ntiles, first, nfirst, queue, stats, warps, nsm, s
#define RF_DECL_RASTER_TW(TW)                                         \
    cudaError_t launch_raster_tw##TW(int kind, RF_RASTER_PARAMS);      \
    cudaError_t launch_raster_any_tw##TW(int kind, RF_RASTER_PARAMS);
RF_DECL_RASTER_TW(8)
RF_DECL_RASTER_TW(16)
RF_DECL_RASTER_TW(32)
RF_DECL_RASTER_TW(64)
#undef RF_DECL_RASTER_TW
// The raster pass: a launch per group, on the streams st[0 .. nst) in turn
// (the caller orders the side streams after and before its own).
cudaError_t launch_raster(uint32_t tile_w, const RasterGroup *groups, uint32_t ng, const JobDev *jobs, uint32_t nj,
                          const DrawDev *draws, const PrimRec *prims, const RasterPrim *rprims, const uint32_t *rows,
                          const uint2 *ent, const uint32_t *mask, const uint2 *segs,
                          const uint2 *list, uint32_t ntiles, const uint32_t *items, uint32_t *counters,
                          StatsDev *stats, uint32_t warps, int nsm, const cudaStream_t *st, uint32_t nst);
// Loads the groups' raster kernels for a tile width: a kernel's first launch in a
// process does so otherwise.
cudaError_t load_raster(uint32_t tile_w, const RasterGroup *groups, uint32_t ng);
cudaError_t launch_fill(uint32_t *color, float *depth, size_t n, uint32_t px, float z,
                        uint32_t flags, int nsm, cudaStream_t s);
// Object culling of the draws with RF_DRAW_CULL_BBOX (sets DrawDev::culled
// and counts into stats[draw.job]).
cudaError_t launch_cull(DrawDev *draws, uint32_t nd, StatsDev *stats, int nsm, cudaStream_t s);
// Line primitives (rf_lines.cu): setup + tile raster of one line draw
// (draws[0], jobs[0]; mask zeroed, queue zeroed).
cudaError_t launch_lines(const DrawDev *draws, const JobDev *jobs, uint32_t nl, const float4 *cpos,
                         const uint8_t *coc, LineRec *recs, uint32_t *mask, uint32_t ntiles,
                         uint32_t *queue, StatsDev *stats, int nsm, cudaStream_t s);
// Depth sort (render.rs:180-182, 209-219; rf_sort.cu).  launch_dsort: the
// key of every clipped triangle -- its draw, then Render::depth (the mean
// clip-space z, prim.rs:21-23) in f32::total_cmp order, ascending or
// descending per its job's depth_sort (0 for jobs without) -- sorted stably,
// so perm[r] is the clipped-order index of the r-th triangle; ptri[p] is the
// input triangle of clipped triangle p.  np = the frame's clipped
// triangles (host-known); scan_scratch holds
// scan_scratch_words(dsort_scan_items(np)) words.
size_t dsort_scratch_bytes(uint32_t np);
uint32_t dsort_scan_items(uint32_t np);
cudaError_t launch_dsort(const DrawDev *draws, uint32_t nd, const JobDev *jobs, uint32_t nt,
                         uint32_t np, const float4 *cpos, const uint32_t *tcnt, const uint32_t *toff,
                         const uint32_t *tpoly, const PolyVert *pool, const uint32_t *counters,
                         uint32_t *perm, uint32_t *ptri, void *scratch, uint32_t *scan_scratch,
                         cudaStream_t s);
// Per-draw clipped-triangle counts only (nout[d]), before np is known.
cudaError_t launch_draw_counts(const DrawDev *draws, uint32_t nd, uint32_t nt, const uint32_t *toff,
                               const uint32_t *counters, uint32_t *nout, cudaStream_t s);
// Writes the GPU's global timer (ns) into *dst when the stream reaches it
// (dst: device memory or page-locked host memory).
cudaError_t launch_stamp(unsigned long long *dst, cudaStream_t s);
// Adds the n per-job stats slots js[0..n) into *total (one block).
cudaError_t launch_stats_fold(const StatsDev *js, uint32_t n, StatsDev *total, cudaStream_t s);
}  // namespace rfk

#endif
