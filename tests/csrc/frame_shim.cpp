// Host build of the frame code (rf_api.cu) against a CUDA runtime that is all
// host memory, for CPU tests of what a frame's buffers hold between frames.
// Copies, fills and launches happen at once.  An allocation takes the address
// freed last, whatever its size was, and holds 0xA5 bytes; the kernels' stand-ins
// do what the frame's contract says of the tile masks: zero when the setup
// pass marks them, zero again once the list pass has read them.
#include <sys/mman.h>

#include <set>
#include <string>

#include "../../retrofire_gb300/csrc/rf_api.cu"

namespace {
constexpr size_t SLOT = 256u << 20;
constexpr int NSLOTS = 256;
char *g_base = nullptr;
int g_next = 0;
int g_fail_event = -1;       // the event that is not made, counted down to (-1: none)
int g_fail_alloc = -1;       // the allocation that fails, counted down to (-1: none)
uint64_t g_null_counters = 0, g_bad_counters = 0;  // zeroing launches without counters; counters of a new context not zero
std::vector<int> g_free;
int g_fail_lists = 0;        // the list pass reports an error this many times
int g_fail_fill = 0;         // ... a fill of more than a few counters
uint32_t g_clipped = 1;      // a sorted frame's clipped triangles per input one
uint64_t g_dirty_words = 0;  // mask words found set when a setup pass began
uint64_t g_setups = 0, g_same_address = 0;
size_t g_size[NSLOTS];       // bytes allocated in each slot
size_t g_host_limit = ~(size_t)0, g_host_bytes = 0;  // largest page-locked allocation allowed; bytes asked for
uint64_t g_bad_draws = 0, g_seen_draws = 0;  // descriptors that reached the device, and wrong ones
uint32_t g_tris = 1;                         // triangles of every draw
const void *g_last_mask = nullptr;
size_t g_last_size = 0;

// The frames' calls: B(egin of a capture), I(nstantiate), U(pload), G(raph
// launch), R(aster launch), L(oad of raster kernels), E(vent that times), a bar after each.
std::string g_log;
float g_trial_ms[4] = {1, 1, 1, 1};  // what the trials of a context take
int g_trial = 0;
std::vector<RasterGroup> g_groups;   // of the last frame
std::set<cudaStream_t> g_streams;    // ... that its groups are on

// Words of the masks and summaries the jobs lay out.
size_t job_words(const JobDev *jobs, uint32_t nj) {
    size_t n = 0;
    for (uint32_t j = 0; j < nj; ++j)
        n = std::max<size_t>(n, jobs[j].sum_base + (size_t)jobs[j].tiles_x * jobs[j].tiles_y * jobs[j].sum_words);
    return n;
}
}  // namespace

extern "C" {
cudaError_t cudaMalloc(void **p, size_t n) {
    if (g_fail_alloc >= 0 && g_fail_alloc-- == 0) return cudaErrorMemoryAllocation;
    if (!g_base) {
        void *m = mmap(nullptr, SLOT * NSLOTS, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
        if (m == MAP_FAILED) return cudaErrorMemoryAllocation;
        g_base = static_cast<char *>(m);
    }
    int slot = g_next;
    if (!g_free.empty()) {
        slot = g_free.back();
        g_free.pop_back();
    } else if (g_next++ == NSLOTS) {
        return cudaErrorMemoryAllocation;
    }
    if (n > SLOT) return cudaErrorMemoryAllocation;
    *p = g_base + SLOT * (size_t)slot;
    g_size[slot] = n;
    memset(*p, 0xA5, n);
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    if (p) g_free.push_back((int)((static_cast<char *>(p) - g_base) / (ptrdiff_t)SLOT));
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) {
    g_host_bytes += n;
    return n <= g_host_limit && (*p = malloc(n)) ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaMallocHost(void **p, size_t n) { return cudaHostAlloc(p, n, 0); }
cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) {
    if (n > 1024 && g_fail_fill) {
        --g_fail_fill;
        return cudaErrorUnknown;
    }
    memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 4; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaEventCreate(cudaEvent_t *e) {  // (2: one that times)
    if (g_fail_event >= 0 && g_fail_event-- == 0) return cudaErrorMemoryAllocation;
    *e = reinterpret_cast<cudaEvent_t>(2);
    return cudaSuccess;
}
cudaError_t event_ok(cudaEvent_t e) { return e ? cudaSuccess : cudaErrorInvalidResourceHandle; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
    const cudaError_t st = cudaEventCreate(e);
    if (!st) *e = reinterpret_cast<cudaEvent_t>(1);
    return st;
}
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
    *ms = g_trial < 4 ? g_trial_ms[g_trial++] : 1.0f;
    return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t e) { return event_ok(e); }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) {
    if (e == reinterpret_cast<cudaEvent_t>(2)) g_log += 'E';
    return event_ok(e);
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) { return event_ok(e); }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t, unsigned long long) {
    g_log += 'I';
    *x = reinterpret_cast<cudaGraphExec_t>(1);
    return cudaSuccess;
}
cudaError_t cudaGraphUpload(cudaGraphExec_t, cudaStream_t) { g_log += 'U'; return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { g_log += 'G'; return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { g_log += 'B'; return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) { *g = nullptr; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
    static uintptr_t n = 0;
    *s = reinterpret_cast<cudaStream_t>(++n);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t e, unsigned) { return event_ok(e); }
}

namespace rfk {
cudaError_t launch_zero(uint32_t *mask, size_t words, bool masks, StatsDev *js, uint32_t njobs, unsigned long long *tacc,
                        uint32_t ntiles, unsigned long long *totals, unsigned long long *marks, uint32_t *counters, int,
                        cudaStream_t) {
    if (!counters) {
        ++g_null_counters;
        return cudaSuccess;
    }
    for (int i = 0; i < RF_CNT_N; ++i) g_bad_counters += counters[i] != 0u;
    if (masks) memset(mask, 0, words * 4);
    memset(js, 0, njobs * sizeof(StatsDev));
    memset(tacc, 0, (size_t)ntiles * 8);
    totals[0] = totals[1] = *marks = 0;
    return cudaSuccess;
}
cudaError_t launch_setup(const DrawDev *, uint32_t, const JobDev *jobs, uint32_t nj, const RasterGroup *, uint32_t,
                         uint32_t, uint32_t, const float4 *, const uint32_t *, const uint32_t *, const uint32_t *,
                         const PolyVert *, PrimRec *, unsigned long long *, uint32_t *, unsigned long long, RasterPrim *,
                         uint2 *, uint32_t *mask, uint32_t *, unsigned long long *, StatsDev *, uint32_t *, int,
                         cudaStream_t, const uint32_t *, const uint32_t *) {
    const size_t n = job_words(jobs, nj);
    for (size_t i = 0; i < n; ++i) g_dirty_words += mask[i] != 0u;
    ++g_setups;
    const size_t size = g_size[(reinterpret_cast<char *>(mask) - g_base) / (ptrdiff_t)SLOT];
    g_same_address += mask == g_last_mask && size > g_last_size;
    g_last_mask = mask;
    g_last_size = size;
    memset(mask, 0xFF, n * 4);  // (all marked)
    return cudaSuccess;
}
cudaError_t launch_lists(const JobDev *jobs, uint32_t nj, uint32_t *mask, uint32_t, uint32_t, const uint2 *,
                         unsigned long long *, const unsigned long long *, uint32_t, uint32_t *, uint32_t *, uint2 *,
                         uint2 *, unsigned long long *, unsigned long long, cudaStream_t) {
    if (g_fail_lists) {
        --g_fail_lists;
        return cudaErrorUnknown;
    }
    memset(mask, 0, job_words(jobs, nj) * 4);
    return cudaSuccess;
}
cudaError_t launch_draw_counts(const DrawDev *d, uint32_t nd, uint32_t, const uint32_t *, const uint32_t *, uint32_t *nout,
                               cudaStream_t) {
    for (uint32_t i = 0; i < nd; ++i) nout[i] = d[i].ntri * g_clipped;
    return cudaSuccess;
}
cudaError_t launch_vertex(const DrawDev *d, uint32_t nd, uint32_t, float4 *, uint8_t *, uint32_t *, int, cudaStream_t) {
    for (uint32_t i = 0; i < nd; ++i)
        g_bad_draws += d[i].tri_base != i * g_tris || d[i].mvp[0] != (float)i || d[i].verts == nullptr;
    g_seen_draws += nd;
    return cudaSuccess;
}
cudaError_t launch_cull(DrawDev *, uint32_t, StatsDev *, int, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_clip(const DrawDev *, uint32_t, uint32_t, const float4 *, const uint8_t *, uint32_t *, uint32_t *,
                        uint32_t *, PolyVert *, uint32_t, uint32_t *, int, cudaStream_t, uint32_t *, bool) { return cudaSuccess; }
cudaError_t launch_fill(uint32_t *, float *, size_t, uint32_t, float, uint32_t, int, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_scan(const uint32_t *, uint32_t *, uint32_t, uint32_t *, uint32_t *, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_dsort(const DrawDev *, uint32_t, const JobDev *, uint32_t, uint32_t, const float4 *, const uint32_t *,
                         const uint32_t *, const uint32_t *, const PolyVert *, const uint32_t *, uint32_t *, uint32_t *,
                         void *, uint32_t *, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_lines(const DrawDev *, const JobDev *, uint32_t, const float4 *, const uint8_t *, LineRec *, uint32_t *,
                         uint32_t, uint32_t *, StatsDev *, int, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_stamp(unsigned long long *, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_raster(uint32_t, const RasterGroup *g, uint32_t ng, const JobDev *, uint32_t, const DrawDev *,
                          const PrimRec *, const RasterPrim *, const uint32_t *, const uint2 *, const uint32_t *,
                          const uint2 *, const uint2 *, uint32_t, const uint32_t *, uint32_t *, StatsDev *, uint32_t, int,
                          const cudaStream_t *st, uint32_t nst) {
    g_log += 'R';
    g_groups.assign(g, g + ng);
    g_streams.clear();
    for (uint32_t i = 0; i < ng; ++i) g_streams.insert(st[i % nst]);
    return cudaSuccess;
}
cudaError_t load_raster(uint32_t, const RasterGroup *, uint32_t) { g_log += 'L'; return cudaSuccess; }
cudaError_t launch_mesh_bbox(const float *, uint32_t, uint32_t, float *, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_stats_fold(const StatsDev *, uint32_t, StatsDev *, cudaStream_t) { return cudaSuccess; }
uint32_t dsort_scan_items(uint32_t) { return 0; }
size_t scan_scratch_words(uint32_t n) { return n / 4096u + 2u; }
size_t dsort_scratch_bytes(uint32_t n) { return (size_t)n * 32u + 4096u; }
}  // namespace rfk

namespace {
// One frame of ndraws draws of one mesh of ntri flat triangles on a w x h
// target; claims: the number of draws the call says it has (the one after the
// last is a bad handle then).
rf_status frame(rf_ctx *ctx, uint32_t ntri, uint32_t w, uint32_t h, int32_t sort, uint32_t ndraws = 1,
                uint32_t claims = 0) {
    std::vector<float> v(9, 0.5f);
    std::vector<uint32_t> idx(3 * (size_t)ntri);
    for (size_t i = 0; i < idx.size(); ++i) idx[i] = (uint32_t)(i % 3);
    g_tris = ntri;
    rf_mesh m = 0;
    rf_target t = 0;
    rf_status st = rf_mesh_upload(ctx, v.data(), 3, 3, 0, idx.data(), ntri, &m);
    if (!st) st = rf_target_create(ctx, w, h, RF_ARGB8888, 1, &t);
    if (!st) {
        std::vector<rf_draw> d(ndraws + 1);
        for (uint32_t i = 0; i < ndraws; ++i) {
            d[i].mesh = m;
            d[i].shader = RF_SHADER_FLAT;
            d[i].uniforms.mvp[0] = (float)i;
        }
        const float vp[16] = {1, 0, 0, 0, 0, 1, 0, 0, 0, 0, 1, 0, 0, 0, 0, 1};
        const rf_context_flags fl{RF_DEPTH_LESS, 1, 1, RF_CULL_BACK, sort};
        st = rf_render_draws(ctx, d.data(), claims ? claims : ndraws, vp, t, &fl, nullptr);
    }
    if (t) rf_target_destroy(ctx, t);
    if (m) rf_mesh_destroy(ctx, m);
    return st;
}
}  // namespace

extern "C" {
// Frames of the given sizes (ntri, w, h, depth_sort, clipped pieces per
// triangle, 1 when the list pass is to fail, 2 when the zeroing of its masks
// is), one after the other on one context.  out: mask words found set at the setup passes, setup passes,
// those whose masks had grown in place; returns the frames that ended in
// another status than expected.
uint32_t shim_frames(const uint32_t *f, uint32_t n, uint64_t out[3]) {
    rf_ctx *ctx = nullptr;
    if (rf_ctx_create(nullptr, &ctx)) return 0xFFFFFFFFu;
    rf_ctx_set_tiling(ctx, 32, 4);
    g_dirty_words = g_setups = g_same_address = 0;
    g_last_mask = nullptr;
    g_last_size = 0;
    uint32_t bad = 0;
    for (uint32_t i = 0; i < n; ++i, f += 6) {
        g_clipped = f[4];
        g_fail_lists = f[5] == 1u;
        g_fail_fill = f[5] == 2u;
        bad += (frame(ctx, f[0], f[1], f[2], (int32_t)f[3]) == RF_OK) != (f[5] == 0u);
    }
    rf_ctx_destroy(ctx);
    out[0] = g_dirty_words;
    out[1] = g_setups;
    out[2] = g_same_address;
    return bad;
}
uint32_t shim_zero_blocks(uint64_t n16, int masks, uint32_t ntiles, int nsm) {
    return rfk::zero_blocks(n16, masks != 0, ntiles, nsm);
}
// Frames of counts[i] draws each on one context, page-locked allocations above
// `limit` bytes refused.  out: wrong descriptors, descriptors, page-locked
// bytes asked for.  Returns the first status that is not RF_OK.
int32_t shim_draws(const uint32_t *counts, uint32_t n, uint64_t limit, uint64_t out[3]) {
    rf_ctx *ctx = nullptr;
    if (rf_ctx_create(nullptr, &ctx)) return -1;
    g_host_limit = limit;
    g_host_bytes = g_bad_draws = g_seen_draws = 0;
    rf_status st = RF_OK;
    for (uint32_t i = 0; i < n && !st; ++i) st = frame(ctx, 1, 64, 64, 0, counts[i]);
    rf_ctx_destroy(ctx);
    g_host_limit = ~(size_t)0;
    out[0] = g_bad_draws;
    out[1] = g_seen_draws;
    out[2] = g_host_bytes;
    return st;
}
// A call of `good` draws, then a bad handle, that claims to have `claims` draws: its
// status, and the page-locked bytes it asked for.
int32_t shim_refused(uint32_t good, uint32_t claims, uint64_t *bytes) {
    rf_ctx *ctx = nullptr;
    if (rf_ctx_create(nullptr, &ctx)) return -1;
    g_host_bytes = 0;
    const rf_status st = frame(ctx, 2, 64, 64, 0, good, claims);
    *bytes = g_host_bytes;
    rf_ctx_destroy(ctx);
    return st;
}
// On a new context, a frame whose k-th allocation fails (its mesh and target
// included), then one that has all it asks for: the first one's status; out: the
// second's, zeroing launches without counters, counters found set.
int32_t shim_alloc_fails(uint32_t k, uint64_t out[3]) {
    rf_ctx *ctx = nullptr;
    if (rf_ctx_create(nullptr, &ctx)) return -1;
    g_null_counters = g_bad_counters = 0;
    g_fail_alloc = (int)k;
    const rf_status st = frame(ctx, 5, 64, 64, 0);
    g_fail_alloc = -1;
    out[0] = frame(ctx, 5, 64, 64, 0);
    out[1] = g_null_counters;
    out[2] = g_bad_counters;
    rf_ctx_destroy(ctx);
    return st;
}
// On a new context, a batch of two raster groups during which the k-th event
// cannot be made, then the same again with nothing failing: the first one's status;
// out: the second's.
int32_t shim_event_fails(uint32_t k, int32_t *out) {
    rf_ctx *ctx = nullptr;
    if (rf_ctx_create(nullptr, &ctx)) return -1;
    rf_ctx_set_tiling(ctx, 32, 4);
    const float v[9] = {};
    const uint32_t idx[3] = {0, 1, 2};
    rf_mesh m = 0;
    rf_target t[2] = {0, 0};
    rf_status st = rf_mesh_upload(ctx, v, 3, 3, 0, idx, 1, &m);
    for (int i = 0; i < 2 && !st; ++i) st = rf_target_create(ctx, 64, 64, RF_ARGB8888, 1, &t[i]);
    if (st) return -1;
    g_tris = 1;
    rf_draw d{};
    d.mesh = m;
    d.shader = RF_SHADER_FLAT;
    rf_job j[2]{};
    for (int i = 0; i < 2; ++i) {
        j[i].target = t[i];
        j[i].ndraws = 1;
        j[i].draws = &d;
        j[i].flags = {i ? RF_DEPTH_GREATER : RF_DEPTH_LESS, 1, 1, RF_CULL_BACK, 0};
    }
    g_fail_event = (int)k;
    st = rf_render_batch(ctx, j, 2, nullptr);
    g_fail_event = -1;
    *out = rf_render_batch(ctx, j, 2, nullptr);
    rf_ctx_destroy(ctx);
    return st;
}
// A batch of n jobs (shader, 1 for the default context or 0, triangles): its raster
// groups as (shader, default context, triangles), the streams they are on and
// the kernels counted; returns the groups, or -1.
int32_t shim_groups(const uint32_t *jobs, uint32_t n, uint32_t *out, uint32_t *streams, uint64_t *kernels) {
    rf_ctx *ctx = nullptr;
    if (rf_ctx_create(nullptr, &ctx)) return -1;
    rf_ctx_set_tiling(ctx, 32, 4);
    std::vector<rf_draw> d(n);
    std::vector<rf_job> j(n);
    const std::vector<float> v(3 * 7, 0.5f);
    g_tris = 0;  // (descriptors not looked at)
    for (uint32_t i = 0; i < n; ++i) {
        const uint32_t *q = jobs + 3 * i;
        std::vector<uint32_t> idx(3 * (size_t)q[2], 0u);
        if (rf_mesh_upload(ctx, v.data(), 3, 4, q[0] == RF_SHADER_FLAT ? 0 : 3, idx.data(), q[2], &d[i].mesh)) return -1;
        if (rf_target_create(ctx, 32, 32, RF_ARGB8888, 1, &j[i].target)) return -1;
        d[i].shader = (int32_t)q[0];
        j[i].ndraws = 1;
        j[i].draws = &d[i];
        j[i].flags = {q[1] ? RF_DEPTH_LESS : RF_DEPTH_GREATER, 1, 1, RF_CULL_BACK, 0};
    }
    if (rf_render_batch(ctx, j.data(), n, nullptr)) return -1;
    rf_ctx_counts(ctx, kernels, nullptr, nullptr);
    rf_ctx_destroy(ctx);
    for (size_t g = 0; g < g_groups.size(); ++g) {
        out[3 * g] = (uint32_t)g_groups[g].kind;
        out[3 * g + 1] = g_groups[g].fast;
        out[3 * g + 2] = g_groups[g].ntri;
    }
    *streams = (uint32_t)g_streams.size();
    return (int32_t)g_groups.size();
}
// n frames of one shape with the tile width picked online; log: their calls.
int32_t shim_trials(uint32_t n, int graphs, int32_t sort, char *log, uint32_t room) {
    rf_ctx *ctx = nullptr;
    if (rf_ctx_create(nullptr, &ctx)) return -1;
    rf_ctx_set_graphs(ctx, graphs);
    g_log.clear();
    rf_status st = RF_OK;
    for (uint32_t i = 0; i < n && !st; ++i) {
        st = frame(ctx, 20, 64, 64, sort);
        g_log += '|';
    }
    rf_ctx_destroy(ctx);
    snprintf(log, room, "%s", g_log.c_str());
    return st;
}
// The tile width picked for a frame whose trials take ms[0..4).
uint32_t shim_pick(const float *ms, int graphs) {
    rf_ctx *ctx = nullptr;
    if (rf_ctx_create(nullptr, &ctx)) return 0;
    rf_ctx_set_graphs(ctx, graphs);
    memcpy(g_trial_ms, ms, sizeof g_trial_ms);
    g_trial = 0;
    for (int i = 0; i < 6; ++i)
        if (frame(ctx, 20, 64, 64, 0)) return 0;
    uint32_t w = 0;
    rf_ctx_last_tiling(ctx, &w, nullptr);
    rf_ctx_destroy(ctx);
    return w;
}
}
