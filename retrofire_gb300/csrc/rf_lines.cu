// rf_lines.cu — line primitives: render() for Edge<usize> (core/src/render/
// prim.rs:41-60): the vertex stage (k_vertex), line clipping (clip.rs:
// 311-348), to_screen, face culling (is_backface is false for an edge), and
// line() (raster.rs:115-173), each pixel a one-pixel scanline into the
// target (target.rs:163-198) with the first vertex's position and varyings.
//
// k_line_setup: one thread per line; clips it, walks its pixels with the
// reference's running sum (stats, and the tiles it touches: a per-tile
// bitmask over the lines, bit order = submission order).
// k_line_raster: a warp per quarter or half of a 32x32 tile (8 or 16 rows, its
// pixels in shared memory unless its lines are few) takes the tile's lines in
// order, 32 at a time, and their steps inside its columns (a line that steps
// along x) or rows, 32 of any lines a pass: a lane's pixel comes from the
// running sum, and lanes that meet in a pixel go in submission order.
#include "rf_raster.cuh"

using namespace rfx;
using namespace rfd;

namespace {

__constant__ float l_planes[6][4] = {
    {0.0f, 0.0f, -1.0f, -1.0f},  // near   (clip.rs:215-222)
    {0.0f, 0.0f, 1.0f, -1.0f},   // far
    {-1.0f, 0.0f, 0.0f, -1.0f},  // left
    {1.0f, 0.0f, 0.0f, -1.0f},   // right
    {0.0f, -1.0f, 0.0f, -1.0f},  // bottom
    {0.0f, 1.0f, 0.0f, -1.0f},   // top
};

__device__ __forceinline__ uint32_t loutcode(const float *p) {
    uint32_t oc = 0;
#pragma unroll
    for (int i = 0; i < 6; ++i) oc |= (dot4(l_planes[i], p) > 0.0f) ? (1u << i) : 0u;
    return oc;
}

struct LV {
    float pos[4];
    float a[RF_MAX_ATTR];
    uint32_t oc;
};

// ClipPlane::intersect (clip.rs:121-145) on one edge.
__device__ bool lintersect(int p, const LV &a, const LV &b, uint32_t na, LV &out) {
    const float d0 = dot4(l_planes[p], a.pos), d1 = dot4(l_planes[p], b.pos);
    if (!(fmul(d0, d1) < 0.0f)) return false;
    const float t = fdiv(-d0, fsub(d1, d0));
#pragma unroll
    for (int c = 0; c < 4; ++c) out.pos[c] = lerp(a.pos[c], b.pos[c], t);
    for (uint32_t c = 0; c < na; ++c) out.a[c] = lerp(a.a[c], b.a[c], t);
    out.oc = loutcode(out.pos);
    return true;
}

__device__ __forceinline__ uint32_t lzdiv_mask(int32_t shader) {
    return shader == RF_K_TEXTURED ? 0x3u : (shader == RF_K_TEX_GOURAUD ? 0x18u : 0u);
}

// Shaded colour of a fragment with varyings v (v[0] = z, v[1..] attributes
// after to_screen), packed in the target's format.
__device__ uint32_t lshade(const DrawDev &dd, const float *v, int32_t fmt) {
    using namespace rfr;
    const Paint d(dd);
    uint32_t c;
    switch (dd.shader) {
        case RF_K_FLAT: c = Kind<RF_K_FLAT>::shade(d, v); break;
        case RF_K_GOURAUD: c = Kind<RF_K_GOURAUD>::shade(d, v); break;
        case RF_K_TEXTURED: c = Kind<RF_K_TEXTURED>::shade(d, v); break;
        case RF_K_TEX_GOURAUD: c = Kind<RF_K_TEX_GOURAUD>::shade(d, v); break;
        default: c = Kind<RF_K_GOURAUD_SRGB>::shade(d, v); break;
    }
    return pack_px(c, pack_selector(fmt));
}

}  // namespace

__global__ void k_line_setup(const DrawDev *__restrict__ draws, const JobDev *__restrict__ jobs,
                             uint32_t nl, const float4 *cpos,
                             const uint8_t *coc, LineRec *__restrict__ recs,
                             uint32_t *__restrict__ mask, StatsDev *__restrict__ stats) {
    rfd::grid_begin();
    const DrawDev &d = draws[0];
    const JobDev &J = jobs[0];
    const uint32_t na = d.nattr, zm = lzdiv_mask(d.shader);
    unsigned long long po = 0, fi = 0, oob = 0;
    for (uint32_t l = blockIdx.x * blockDim.x + threadIdx.x; l < nl; l += gridDim.x * blockDim.x) {
        LineRec R{};
        LV e[2];
        for (int k = 0; k < 2; ++k) {
            const uint32_t vi = d.idx[2 * (size_t)l + k];
            const float4 p = cpos[vi];
            e[k].pos[0] = p.x; e[k].pos[1] = p.y; e[k].pos[2] = p.z; e[k].pos[3] = p.w;
            e[k].oc = coc[vi];
            const float *src = d.verts + (size_t)vi * d.stride + d.pos_dim;
            for (uint32_t c = 0; c < RF_MAX_ATTR; ++c) e[k].a[c] = c < na ? src[c] : 0.0f;
        }
        bool keep = (e[0].oc & e[1].oc) == 0;  // both outside one plane: dropped
        if (keep && (e[0].oc | e[1].oc)) {
            for (int p = 0; p < 6; ++p) {
                const bool a_in = (e[0].oc & (1u << p)) == 0, b_in = (e[1].oc & (1u << p)) == 0;
                if (!a_in && !b_in) {
                    keep = false;
                    break;
                }
                LV v;
                if (lintersect(p, e[0], e[1], na, v)) {
                    if (a_in) e[1] = v;
                    else if (b_in) e[0] = v;
                }
            }
        }
        // to_screen (prim.rs:62-88): (x/w, y/w, 1/w) through the viewport,
        // attributes z_div'd where the shader's types divide.
        float s[2][3], at[2][RF_MAX_ATTR];
        if (keep) {
            for (int k = 0; k < 2; ++k) {
                const float w = e[k].pos[3];
                const float ndc[4] = {fdiv(e[k].pos[0], w), fdiv(e[k].pos[1], w), fdiv(1.0f, w), 1.0f};
                s[k][0] = dot4(J.vp + 0, ndc);
                s[k][1] = dot4(J.vp + 4, ndc);
                s[k][2] = dot4(J.vp + 8, ndc);
                for (uint32_t c = 0; c < RF_MAX_ATTR; ++c)
                    at[k][c] = c < na ? (((zm >> c) & 1u) ? fdiv(e[k].a[c], w) : e[k].a[c]) : 0.0f;
            }
            if (J.face_cull == RF_K_CULL_FRONT) keep = false;  // face_cull(false)
        }
        if (keep) {
            po += 1;
            // raster.rs:121-173 line(): v0 the upper end, then for a wide
            // line the left end (dx, dy keep their values).
            int i0 = 0, i1 = 1;
            if (s[0][1] > s[1][1]) { i0 = 1; i1 = 0; }
            const float dx = fsub(s[i1][0], s[i0][0]), dy = fsub(s[i1][1], s[i0][1]);
            const bool wide = fabsf(dx) > dy;
            if (wide && dx < 0.0f) { const int t = i0; i0 = i1; i1 = t; }
            uint64_t b, e2;
            float s0, dd;
            if (wide) {
                const float x0 = round_up_to_half(s[i0][0]), x1 = round_up_to_half(s[i1][0]);
                dd = fdiv(dy, dx);
                s0 = fadd(s[i0][1], fmul(dd, fsub(x0, s[i0][0])));
                b = as_usize(x0);
                e2 = as_usize(x1);
            } else {
                const float y0 = round_up_to_half(s[i0][1]), y1 = round_up_to_half(s[i1][1]);
                dd = fdiv(dx, dy);
                s0 = fadd(s[i0][0], fmul(dd, fsub(y0, s[i0][1])));
                b = as_usize(y0);
                e2 = as_usize(y1);
            }
            const uint64_t n = e2 > b ? e2 - b : 0u;
            if (n > RF_LINE_MAX_SPAN) {
                oob += 1;  // out of the supported range: counted, not drawn
            } else if (n) {
                float v[RF_NC];
                v[0] = s[i0][2];
                for (uint32_t c = 0; c < RF_MAX_ATTR; ++c) v[1 + c] = at[i0][c];
                R.live = 1;
                R.wide = wide ? 1u : 0u;
                R.begin = b;
                R.n = (uint32_t)n;
                R.s0 = s0;
                R.d = dd;
                R.z = v[0];
                R.color = J.color_write ? lshade(d, v, J.pixfmt) : 0u;
                // The pixels with the running sum, for the stats and tiles.
                float val = s0;
                uint32_t last = 0xFFFFFFFFu;
                for (uint64_t k = 0; k < n; ++k) {
                    const uint64_t x = wide ? b + k : as_usize(val);
                    const uint64_t y = wide ? as_usize(val) : b + k;
                    val = fadd(val, dd);
                    if (y >= J.h) {
                        oob += 1;
                        continue;
                    }
                    fi += 1;
                    if (x >= J.w) {
                        oob += 1;
                        continue;
                    }
                    const uint32_t tile = (uint32_t)(y / RF_TILE_H) * J.tiles_x + (uint32_t)(x / RF_TILE_H);
                    if (tile != last) {
                        atomicOr(mask + (size_t)tile * J.mask_words + (l >> 5), 1u << (l & 31));
                        last = tile;
                    }
                }
            }
        }
        recs[l] = R;
    }
    warp_add_u64(&stats->prims_o, po, true);
    warp_add_u64(&stats->verts_o, 3ull * po, true);
    warp_add_u64(&stats->frags_i, fi, true);
    warp_add_u64(&stats->oob, oob, true);
}

// The k-step running sum from s: one add after the other up to RF_LINE_STEP
// steps (4 cycles each; a wireframe's lines are mostly shorter, and so are a
// line's steps in a tile), else the exact jump.
#define RF_LINE_STEP 64u
__device__ __forceinline__ float line_step(float s, float d, uint32_t k) {
    if (k > RF_LINE_STEP) return jump(s, d, k);
#pragma unroll 1
    for (; k >= 4u; k -= 4u) s = fadd(fadd(fadd(fadd(s, d), d), d), d);
#pragma unroll
    for (uint32_t i = 0; i < 3; ++i)
        if (i < k) s = fadd(s, d);
    return s;
}

// Leaves out steps of a line (n of them, the first at R.begin with the value
// R.s0) whose pixels miss the rows (columns) [a0, a1): those the line, as one,
// is more than a pixel away from.  |d| <= 1 and n <= 32, so 32 additions near
// the target are off by far less; below 0 a step draws in row (column) 0.
__device__ __forceinline__ void line_trim(LineRec &R, uint32_t &n, uint32_t a0, uint32_t a1) {
    if (!(fabsf(R.s0) < 1e6f)) return;
    const float lo = a0 ? (float)a0 - 1.0f : -1e7f, hi = (float)a1 + 1.0f, last = (float)n * R.d + R.s0;
    if (fmaxf(R.s0, last) < lo || fminf(R.s0, last) > hi) {
        n = 0;
        return;
    }
    // the steps that enter and leave [lo, hi], moved apart by one
    const float in = R.d > 0.0f ? lo : hi, out = R.d > 0.0f ? hi : lo, r = fdiv(1.0f, R.d);
    const uint32_t k0 = (uint32_t)fminf(fmaxf((in - R.s0) * r - 1.0f, 0.0f), (float)n);
    const uint32_t k1 = (uint32_t)fminf(fmaxf((out - R.s0) * r + 2.0f, 0.0f), (float)n);
    if (!(fabsf(R.d) > 1e-6f) || (k0 == 0u && k1 == n)) return;  // (too flat to cross: every step)
    R.s0 = line_step(R.s0, R.d, k0);
    R.begin += k0;
    n = k1 > k0 ? k1 - k0 : 0u;
}

#define RF_LINE_WARPS 4
#define RF_LINE_PITCH 33u  // words per tile row in shared memory (odd: steep lines hit different banks)
// Bound by the latencies of the fullest tiles (up to 200 lines of a wireframe of
// 12,416 at 1280x720): one line a pass, a lane per column or row, each line's
// record and pixels waited for in turn, took 117 us there.  With a batch's
// records loaded together, the pixels in shared memory and short lines sharing
// a pass 65, and with four warps a tile, ROWS rows each, 31 (each reads all of
// the tile's mask, which is in L2).  The running sum is worked out once a line
// and part, at its first step there, and stepped on from that (with a jump a
// pixel 30,000 lines of up to 3,000 px took 4.0 ms on 320 x 240, 2.7 ms one line
// a pass; now 1.3), and only for the steps that can reach the part's rows.
// Parts with few lines, which are most of a large target's, draw in place: moved
// through shared memory 30,000 lines of up to 20 px on 3840 x 2160 took 210 us,
// now 149.
template <uint32_t ROWS>  // tile rows a warp draws
__global__ void __launch_bounds__(RF_LINE_WARPS * 32)
k_line_raster(const JobDev *__restrict__ jobs, const LineRec *recs,
              const uint32_t *mask, uint32_t ntiles, uint32_t *__restrict__ queue,
              StatsDev *__restrict__ stats) {
    rfd::grid_begin();
    constexpr uint32_t FULL = 0xFFFFFFFFu;
    __shared__ uint32_t s_col[RF_LINE_WARPS][ROWS * RF_LINE_PITCH];
    __shared__ float s_dep[RF_LINE_WARPS][ROWS * RF_LINE_PITCH];
    __shared__ LineRec s_rec[RF_LINE_WARPS][32];
    __shared__ uint32_t s_pend[RF_LINE_WARPS][64];  // the tile's lines found, not drawn yet
    __shared__ uint2 s_item[RF_LINE_WARPS][32];  // per line of the batch with steps here: its lane, first item
    const JobDev &J = jobs[0];
    const uint32_t lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const uint32_t below = (1u << lane) - 1u, upto = below | (1u << lane);
    uint32_t *col = s_col[wib];
    float *dep = s_dep[wib];
    const bool has_depth = J.depth != nullptr, color_write = J.color_write != 0;
    const bool depth_write = has_depth && J.depth_write != 0;
    const int32_t test = has_depth ? J.depth_test : RF_K_DEPTH_NONE;
    unsigned long long fo = 0;
    for (;;) {
        uint32_t part = 0;
        if (lane == 0) part = atomicAdd(queue, 1u);
        part = __shfl_sync(FULL, part, 0);
        const uint32_t tile = part / (RF_TILE_H / ROWS);
        if (tile >= ntiles) break;
        const uint32_t ty = tile / J.tiles_x, tx = tile - ty * J.tiles_x;
        const uint32_t tx0 = tx * RF_TILE_H, tx1 = min(tx0 + RF_TILE_H, J.w);
        const uint32_t ty0 = ty * RF_TILE_H + part % (RF_TILE_H / ROWS) * ROWS;
        if (ty0 >= J.h) continue;
        const uint32_t ty1 = min(ty0 + ROWS, J.h);
        const uint32_t *tm = mask + (size_t)tile * J.mask_words;
        bool loaded = false;
        // The tile's lines in order: 32 mask words at a time (the next four
        // rounds' already loaded), their set bits on to the pending list, which is
        // drawn 32 lines at a time.
        const auto words = [&](uint32_t w) { return w + lane < J.mask_words ? tm[w + lane] : 0u; };
        uint32_t next[4] = {words(0), words(32), words(64), words(96)};
        uint32_t word = 0, incl = 0, nlines = 0, lb = 0, wb = 0, pend = 0;
        for (bool last = false; !last;) {
            if (lb >= nlines) {
                while (wb < J.mask_words && !__any_sync(FULL, next[0] != 0u)) {  // (no lines in these)
                    wb += 32u;
                    next[0] = next[1];
                    next[1] = next[2];
                    next[2] = next[3];
                    next[3] = words(wb + 96u);
                }
                last = wb >= J.mask_words;
                word = last ? 0u : next[0];
                incl = __popc(word);
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(FULL, incl, o);
                    if (lane >= (uint32_t)o) incl += y;
                }
                nlines = __shfl_sync(FULL, incl, 31);
                lb = 0;
                wb += 32u;
                next[0] = next[1];
                next[1] = next[2];
                next[2] = next[3];
                next[3] = words(wb + 96u);
            }
            if (lb < nlines) {
                const uint32_t k = lb + lane;
                const uint32_t L = lane_of(incl, k);
                const uint32_t wl = __shfl_sync(FULL, word, L);
                const uint32_t ex = __shfl_sync(FULL, incl - __popc(word), L);
                if (k < nlines)
                    s_pend[wib][pend + lane] = (wb - 32u + L) * 32u + nth_bit(wl, k - ex + 1u);
                pend += min(nlines - lb, 32u);
                lb += 32u;
            }
            __syncwarp();
            if (pend == 0u || (pend < 32u && !last)) continue;
            {
                // (the part's only batch: its pixels are drawn where they lie)
                const bool direct = last && !loaded && pend <= 32u;
                if (!loaded && !direct) {
                    loaded = true;
#pragma unroll 8
                    for (uint32_t r = 0; r < ROWS; ++r)
                        if (ty0 + r < ty1 && tx0 + lane < tx1) {
                            const size_t i = (size_t)(ty0 + r) * J.w + tx0 + lane;
                            col[r * RF_LINE_PITCH + lane] = J.color[i];
                            if (has_depth) dep[r * RF_LINE_PITCH + lane] = J.depth[i];
                        }
                }
                const uint32_t here = min(pend, 32u);
                const uint32_t line = lane < here ? s_pend[wib][lane] : 0u;
                const uint32_t left = s_pend[wib][32u + lane];  // (past pend: not used)
                __syncwarp();
                s_pend[wib][lane] = left;
                pend -= here;
                uint32_t n = 0;  // this line's steps in the tile's columns (rows)
                if (lane < here) {
                    LineRec R = recs[line];
                    const uint64_t t0 = R.wide ? tx0 : ty0, t1 = R.wide ? tx1 : ty1;
                    const uint64_t a = max(R.begin, t0), b = min(R.begin + R.n, t1);
                    if (a < b) {
                        n = (uint32_t)(b - a);
                        R.s0 = line_step(R.s0, R.d, (uint32_t)(a - R.begin));
                        R.begin = a;
                        line_trim(R, n, R.wide ? ty0 : tx0, R.wide ? ty1 : tx1);
                        s_rec[wib][lane] = R;
                    }
                }
                uint32_t items = n;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(FULL, items, o);
                    if (lane >= (uint32_t)o) items += y;
                }
                const uint32_t total = __shfl_sync(FULL, items, 31), at = items - n;
                const uint32_t nz = __ballot_sync(FULL, n != 0u);
                // (packed: the table's entries are the lines with steps here)
                if (n) s_item[wib][__popc(nz & below)] = make_uint2(lane, at);
                __syncwarp();
#pragma unroll 1
                for (uint32_t base = 0; base < total; base += 32u) {
                    const uint32_t starts = __reduce_or_sync(FULL, n && at - base < 32u ? 1u << (at - base) : 0u);
                    const uint32_t before = __popc(__ballot_sync(FULL, n && at < base));
                    uint32_t idx = 0xFFFFFFFFu, color = 0;
                    float z = 0.0f;
                    if (base + lane < total) {
                        const uint2 it = s_item[wib][before + __popc(starts & upto) - 1u];
                        const LineRec &R = s_rec[wib][it.x];
                        const uint32_t step = base + lane - it.y;
                        const uint64_t along = R.begin + step, across = as_usize(line_step(R.s0, R.d, step));
                        const uint64_t x = R.wide ? along : across, y = R.wide ? across : along;
                        if (x >= tx0 && x < tx1 && y >= ty0 && y < ty1) {
                            idx = ((uint32_t)y - ty0) * RF_LINE_PITCH + ((uint32_t)x - tx0);
                            color = R.color;
                            z = R.z;
                        }
                    }
                    const uint32_t rank = __popc(__match_any_sync(FULL, idx == 0xFFFFFFFFu ? ~lane : idx) & below);
                    const uint32_t rounds = __reduce_max_sync(FULL, rank);
                    for (uint32_t r = 0; r <= rounds; ++r) {
                        if (idx != 0xFFFFFFFFu && rank == r) {
                            const uint32_t py = idx / RF_LINE_PITCH, px = idx - py * RF_LINE_PITCH;
                            const size_t at = direct ? (size_t)(ty0 + py) * J.w + tx0 + px : idx;
                            uint32_t *pc = direct ? J.color : col;
                            float *pd = direct ? J.depth : dep;
                            bool pass = true;
                            const float cur = has_depth ? pd[at] : 0.0f;
                            switch (test) {  // ctx.rs:86-89
                                case RF_K_DEPTH_NONE: pass = true; break;
                                case RF_K_DEPTH_LESS: pass = cur < z; break;
                                case RF_K_DEPTH_EQUAL: pass = cur == z; break;
                                default: pass = cur > z; break;
                            }
                            if (pass) {
                                if (color_write) {
                                    pc[at] = color;
                                    fo += 1;
                                }
                                if (depth_write) pd[at] = z;
                            }
                        }
                        __syncwarp();  // (these pixels before the next round's tests)
                    }
                }
            }
        }
        if (loaded) {
#pragma unroll 8
            for (uint32_t r = 0; r < ROWS; ++r)
                if (ty0 + r < ty1 && tx0 + lane < tx1) {
                    const size_t i = (size_t)(ty0 + r) * J.w + tx0 + lane;
                    if (color_write) J.color[i] = col[r * RF_LINE_PITCH + lane];
                    if (depth_write) J.depth[i] = dep[r * RF_LINE_PITCH + lane];
                }
            __syncwarp();
        }
    }
    warp_add_u64(&stats->frags_o, fo, true);
}

namespace rfk {

cudaError_t launch_lines(const DrawDev *draws, const JobDev *jobs, uint32_t nl, const float4 *cpos,
                         const uint8_t *coc, LineRec *recs, uint32_t *mask, uint32_t ntiles,
                         uint32_t *queue, StatsDev *stats, int nsm, cudaStream_t s) {
    if (nl == 0) return cudaSuccess;
    const uint32_t blocks = min((nl + 127) / 128, (uint32_t)nsm * 8);
    RF_NEXT(k_line_setup, blocks, 128, 0, s, draws, jobs, nl, cpos, coc, recs, mask, stats);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    // Quarters of a tile while those of the target are about as many as the warps
    // that are resident, else halves: lines of up to 3,000 px, 30,000 on 1280 x
    // 720 (920 tiles) 669 us in quarters and 836 in halves, on 1920 x 1080 (2,040)
    // 818 and 769, on 3840 x 2160 1,313 and 1,067.
    const bool quarters = ntiles <= (uint32_t)nsm * 8;
    auto raster = quarters ? k_line_raster<RF_TILE_H / 4> : k_line_raster<RF_TILE_H / 2>;
    const uint32_t parts = ntiles * (quarters ? 4u : 2u);
    const uint32_t rblocks = min((parts + RF_LINE_WARPS - 1) / RF_LINE_WARPS, (uint32_t)nsm * 8);
    RF_NEXT(raster, rblocks, RF_LINE_WARPS * 32, 0, s, jobs, recs, mask, ntiles, queue, stats);
    return cudaGetLastError();
}

}  // namespace rfk
