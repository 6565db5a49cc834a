// rf_raster.cuh — the tile rasteriser (k_raster), included by one
// translation unit per tile width (rf_raster_tw*.cu) so the specialised
// kernels compile in parallel.
#ifndef RF_RASTER_CUH
#define RF_RASTER_CUH

#include <cuda_runtime.h>

#include <mutex>

#include "rf_device.cuh"

// ---------------------------------------------------------------------------
// K4: tile rasteriser.
// A warp owns one tile of RF_TILE_H rows x TW columns (or a row slice of a
// crowded one) at a time.  Colour and depth sit in shared memory column-major
// (word x*32 + row).  The warp takes the tile's triangles from its list
// (k_tile_lists) in submission order, 32 at a time on a table, and draws their
// scanlines -- the items -- in one of two ways:
//   by row   lane r walks row r's triangles, one a round; a round's spans lie
//            on different rows, so every pixel sees its fragments in order
//            without a test.  The spans are cut into 8-pixel segments, the
//            ones the depths hide are dropped, and the rest queue up so that
//            full warps draw them.  For triangles of many rows.
//   packed   32 items a pass, a lane each, whatever triangles they belong to;
//            a span that meets an earlier one of its row waits for it.  For
//            triangles of few rows, which would leave most rows' lanes idle.
// An item starts from its row record (the reference's own running sums: the
// clipped span and the varyings at its first fragment), copied to shared
// memory one round ahead (cp.async); a span that starts left of the tile is
// stepped to it.  Then it steps pixel by pixel like Iter::next.
// What bounds it: the chain of dependent instructions of each warp (16 warps
// per SM, 38 % of issue slots), so what counts is instructions per triangle:
// one warp pass per triangle -- lane = row, most lanes idle on small
// triangles -- measured 478 us on the 500 k-triangle grid at 1080p (now 80 at
// width 8), 337 us on 10 k instanced cubes (85), 2.40 ms on 64 uneven scenes
// (0.52) and 236 us on 100 k triangles of 1..10^4 px^2 (163 at width 16).
// The loop's code has to stay small: with every helper inlined (8,000
// instructions) warps waited on instruction fetch as long as they worked.
// A tile of whole 32-column blocks goes back to HBM through the copy engine
// (cp.async.bulk, one 128-byte row per lane).
// ---------------------------------------------------------------------------
namespace rfr {
using namespace rfx;
using namespace rfd;

// IntoPixel (pixfmt.rs:76-103) of a Color4 packed r | g << 8 | b << 16 |
// a << 24, as one byte permutation: the selector of each format puts the
// channels where the format wants them (XRGB8888's top byte is zero).
__host__ __device__ constexpr uint32_t pack_selector(int32_t fmt) {
    return fmt == RF_K_ARGB8888 ? 0x3012u : fmt == RF_K_XRGB8888 ? 0x4012u : fmt == RF_K_RGBA8888 ? 0x0123u : 0x2103u;
}
__device__ __forceinline__ uint32_t pack_px(uint32_t c, uint32_t sel) { return __byte_perm(c, 0u, sel); }
// The same pixel straight from the channel bytes r, g, b (each 0..255 in a
// 32-bit word): the byte selector over (r | g << 8, b | 0xFF00) -- byte k of
// the Color4 word is byte {0, 1, 4, 5}[k] there, and byte 2 is a zero.
__host__ __device__ constexpr uint32_t rgb_selector(uint32_t sel) {
    uint32_t out = 0;
    for (int i = 0; i < 4; ++i) {
        const uint32_t n = (sel >> (4 * i)) & 0xFu;
        out |= (n == 0u ? 0u : n == 1u ? 1u : n == 2u ? 4u : n == 3u ? 5u : 2u) << (4 * i);
    }
    return out;
}
static_assert(rgb_selector(0x3012u) == 0x5014u && rgb_selector(0x4012u) == 0x2014u &&
                  rgb_selector(0x0123u) == 0x0145u && rgb_selector(0x2103u) == 0x4105u,
              "pixel selectors over the channel bytes");
__device__ __forceinline__ uint32_t pack_rgb(uint32_t r, uint32_t g, uint32_t b, uint32_t rsel) {
    return __byte_perm(__byte_perm(r, g, 0x1140u), b | 0xFF00u, rsel);
}

__device__ __forceinline__ uint32_t to_color4(float r, float g, float b) {
    // color.rs:253-263: (256 * c) as u8, alpha 0xFF.
    return as_u8(fmul(256.0f, r)) | (as_u8(fmul(256.0f, g)) << 8) | (as_u8(fmul(256.0f, b)) << 16) |
           0xFF000000u;
}

// What shading reads of a draw, copied to registers once per span (lanes of
// one pass may be at different draws).
struct Paint {
    const uint32_t *tex;
    uint32_t tw, th, flat_rgba;
    int32_t sampler;
    __device__ __forceinline__ explicit Paint(const DrawDev &d)
        : tex(d.tex), tw(d.tw), th(d.th), flat_rgba(d.flat_rgba), sampler(d.sampler) {}
};

__device__ __forceinline__ uint32_t sample_tex(const Paint &d, float tu, float tv) {
    const float w = (float)d.tw, h = (float)d.th;
    uint32_t u, v;
    if (d.sampler == RF_K_REPEAT_POT) {  // tex.rs:240-266
        u = (uint32_t)as_i32(ffloor(fmul(w, tu))) & (d.tw - 1u);
        v = (uint32_t)as_i32(ffloor(fmul(h, tv))) & (d.th - 1u);
    } else if (d.sampler == RF_K_CLAMP) {  // tex.rs:272-304
        float su = fmul(tu, w), sv = fmul(tv, h);
        const float wm = fsub(w, 1.0f), hm = fsub(h, 1.0f);
        su = su < 0.0f ? 0.0f : (su > wm ? wm : su);
        sv = sv < 0.0f ? 0.0f : (sv > hm ? hm : sv);
        u = as_u32(ffloor(su));
        v = as_u32(ffloor(sv));
    } else {  // SamplerOnce (tex.rs:313-357), index clamped instead of panicking
        u = min(as_u32(fmul(w, tu)), d.tw - 1u);
        v = min(as_u32(fmul(h, tv)), d.th - 1u);
    }
    return __ldg(d.tex + (size_t)v * d.tw + u);
}

template <int KIND>
struct Kind {
    static constexpr int NC = KIND == RF_K_FLAT ? 1
                            : KIND == RF_K_TEXTURED ? 3
                            : KIND == RF_K_TEX_GOURAUD ? 6 : 4;
    static constexpr bool TEXTURED = KIND == RF_K_TEXTURED || KIND == RF_K_TEX_GOURAUD;
    // The texel a fragment samples (textured kinds; any varyings give an
    // in-range index), then the colour from it: shade() split in two so
    // several fragments' texel loads can be in flight together.
    __device__ static __forceinline__ uint32_t texel(const Paint &d, const float *v) {
        if constexpr (KIND == RF_K_TEXTURED) return sample_tex(d, fdiv(v[1], v[0]), fdiv(v[2], v[0]));
        else if constexpr (KIND == RF_K_TEX_GOURAUD) return sample_tex(d, fdiv(v[4], v[0]), fdiv(v[5], v[0]));
        else return 0u;
    }
    __device__ static __forceinline__ uint32_t from_texel(uint32_t t, const float *v) {
        if constexpr (KIND == RF_K_TEX_GOURAUD) {
            // (a power of two: the product is the quotient, exactly)
            const float tr = fmul((float)(t & 0xFFu), 1.0f / 256.0f);
            const float tg = fmul((float)((t >> 8) & 0xFFu), 1.0f / 256.0f);
            const float tb = fmul((float)((t >> 16) & 0xFFu), 1.0f / 256.0f);
            return to_color4(fmul(tr, v[1]), fmul(tg, v[2]), fmul(tb, v[3]));
        } else {
            return t;
        }
    }
    // shade() packed into the target's pixel format (sel: pack_selector,
    // rsel: rgb_selector of it).
    __device__ static __forceinline__ uint32_t shade_px(const Paint &d, const float *v, uint32_t sel,
                                                        uint32_t rsel) {
        if constexpr (KIND == RF_K_GOURAUD) {
            // color.rs:253-263 as in to_color4, the bytes permuted at once
            return pack_rgb(as_u8(fmul(256.0f, v[1])), as_u8(fmul(256.0f, v[2])), as_u8(fmul(256.0f, v[3])), rsel);
        } else {
            return pack_px(shade(d, v), sel);
        }
    }
    __device__ static __forceinline__ uint32_t shade(const Paint &d, const float *v) {
        if constexpr (KIND == RF_K_FLAT) {
            return d.flat_rgba;
        } else if constexpr (KIND == RF_K_GOURAUD) {
            return to_color4(v[1], v[2], v[3]);
        } else if constexpr (KIND == RF_K_TEXTURED) {
            // Scanline::fragments: var.z_div(pos.z) (raster.rs:60-69)
            return sample_tex(d, fdiv(v[1], v[0]), fdiv(v[2], v[0]));
        } else if constexpr (KIND == RF_K_TEX_GOURAUD) {
            return from_texel(texel(d, v), v);
        } else {  // GOURAUD_SRGB: Color3f<LinRgb>::to_srgb (color.rs:383-392)
            const float ig = fdiv(1.0f, 2.2f);
            return to_color4(powf(v[1], ig), powf(v[2], ig), powf(v[3], ig));
        }
    }
};

// Depth bounds of the FAST path: per lane, the minimum current depth of each
// RF_SEG-pixel segment of its tile row (shared memory, word s*32 + lane).
// Under the Less test with depth writes a pixel's depth only grows, so a
// stored minimum stays a lower bound until it is refreshed.
#define RF_SEG 8

struct TileCtx {
    uint32_t *scol;
    float *sdep;
    float *smin;
    uint32_t row;     // the tile row this lane is at: its own, or its item's
    uint32_t y;       // the target row of tile row `lane`
    uint32_t tx0;     // first column of the tile
    uint32_t tx1;     // one past the last column of the tile inside the target
    bool row_ok;
    bool has_depth;
    int32_t depth_test;
    bool color_write, keep_depth;  // keep_depth: the target has depth and it is written
    bool no_test;     // every fragment passes
    uint32_t fmt;     // pack_selector of the target's pixel format
    uint32_t rfmt;    // rgb_selector of fmt
    unsigned long long frags_o;
};

template <int KIND>
struct PreNC {
    static constexpr int NC = KIND == RF_K_ANY ? RF_NC : Kind<KIND == RF_K_ANY ? 0 : KIND>::NC;
    static constexpr int NP = (NC + 1) / 2;  // pairs of components
};
__host__ __device__ constexpr uint32_t row_words(int nc) { return 1u + (uint32_t)nc; }
__device__ __forceinline__ uint32_t kind_nc(uint32_t kind) {
    return kind == RF_K_FLAT ? 1u : kind == RF_K_TEXTURED ? 3u : kind == RF_K_TEX_GOURAUD ? 6u : 4u;
}


template <int KIND>
__device__ __forceinline__ uint32_t shade_any(uint32_t kind, const Paint &d, const float *v, uint32_t sel,
                                              uint32_t rsel) {
    if constexpr (KIND != RF_K_ANY) {
        return Kind<KIND == RF_K_ANY ? 0 : KIND>::shade_px(d, v, sel, rsel);
    } else {
        switch (kind) {
            case RF_K_FLAT: return Kind<RF_K_FLAT>::shade_px(d, v, sel, rsel);
            case RF_K_GOURAUD: return Kind<RF_K_GOURAUD>::shade_px(d, v, sel, rsel);
            case RF_K_TEXTURED: return Kind<RF_K_TEXTURED>::shade_px(d, v, sel, rsel);
            case RF_K_TEX_GOURAUD: return Kind<RF_K_TEX_GOURAUD>::shade_px(d, v, sel, rsel);
            default: return Kind<RF_K_GOURAUD_SRGB>::shade_px(d, v, sel, rsel);
        }
    }
}

// U fragments of one scanline into the tile (raster.rs:60-69, target.rs:
// 163-198), those before `end` of them: v = the varyings of the fragment at
// word idx of the tile, as pairs stepped two at a time (each half of
// add.rn.f32x2 rounds as the single addition).  U > 1: the depths are
// loaded together (this lane alone writes these pixels meanwhile), and so
// are the texels; a load past `end` stays inside the warp's area.
// Advances idx and v; returns how many passed (FAST).
template <int KIND, bool FAST, int U>
__device__ __forceinline__ uint32_t px_group(TileCtx &T, const Paint &d, uint32_t kind, float2 *v, const float2 *dv,
                                             uint32_t &idx, uint32_t end) {
    constexpr int NP = PreNC<KIND>::NP;
    constexpr int K1 = KIND == RF_K_ANY ? 0 : KIND;
    float cur[U];
    bool p[U];
    float w[U][2 * NP];
    float2 x[NP];
#pragma unroll
    for (int u = 0; u < U; ++u) cur[u] = FAST || T.has_depth ? T.sdep[idx + u * RF_TILE_H] : 0.0f;
#pragma unroll
    for (int c = 0; c < NP; ++c) x[c] = v[c];
#pragma unroll
    for (int u = 0; u < U; ++u) {
#pragma unroll
        for (int c = 0; c < NP; ++c) {
            w[u][2 * c] = x[c].x;
            w[u][2 * c + 1] = x[c].y;
            x[c] = __fadd2_rn(x[c], dv[c]);
        }
        const bool in = U == 1 || idx + u * RF_TILE_H < end;
        if constexpr (FAST) {
            p[u] = in && cur[u] < w[u][0];  // ctx.rs:86-89 with Some(Less)
        } else {
            // ctx.rs:86-89, without branches
            const bool lt = cur[u] < w[u][0], eq = cur[u] == w[u][0], gt = cur[u] > w[u][0];
            const bool pass = T.depth_test == RF_K_DEPTH_LESS ? lt : T.depth_test == RF_K_DEPTH_EQUAL ? eq : gt;
            p[u] = in && (T.no_test || pass);
        }
    }
#pragma unroll
    for (int c = 0; c < NP; ++c) v[c] = x[c];
    uint32_t nout = 0;
    if constexpr (FAST && U > 1 && KIND != RF_K_ANY && Kind<K1>::TEXTURED) {
        uint32_t t[U];
#pragma unroll
        for (int u = 0; u < U; ++u) t[u] = p[u] ? Kind<K1>::texel(d, w[u]) : 0u;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (p[u]) {
                T.scol[idx + u * RF_TILE_H] = pack_px(Kind<K1>::from_texel(t[u], w[u]), T.fmt);
                T.sdep[idx + u * RF_TILE_H] = w[u][0];
                ++nout;
            }
    } else if constexpr (U > 1 && (KIND == RF_K_FLAT || KIND == RF_K_GOURAUD)) {
        // A few instructions that read no memory: every pixel's colour is
        // computed and only the stores depend on the depth test.
        uint32_t k[U];
#pragma unroll
        for (int u = 0; u < U; ++u) k[u] = Kind<K1>::shade_px(d, w[u], T.fmt, T.rfmt);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (FAST ? p[u] : p[u] && T.color_write) T.scol[idx + u * RF_TILE_H] = k[u];
            if (FAST ? p[u] : p[u] && T.keep_depth) T.sdep[idx + u * RF_TILE_H] = w[u][0];
            nout += (FAST ? p[u] : p[u] && T.color_write) ? 1u : 0u;
        }
    } else {
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (p[u]) {
                if (FAST || T.color_write) {
                    T.scol[idx + u * RF_TILE_H] = shade_any<KIND>(kind, d, w[u], T.fmt, T.rfmt);
                    ++nout;
                }
                if (FAST || T.keep_depth) T.sdep[idx + u * RF_TILE_H] = w[u][0];
            }
    }
    idx += U * RF_TILE_H;
    return nout;
}

// FAST path: the minimum current depth of segment s of the lane's row.
__device__ __forceinline__ void seg_refresh(TileCtx &T, uint32_t s) {
    const uint32_t base = s * RF_SEG * RF_TILE_H + T.row;
    float m = T.sdep[base];
#pragma unroll
    for (uint32_t x = 1; x < RF_SEG; ++x) m = fminf(m, T.sdep[base + x * RF_TILE_H]);
    T.smin[s * RF_TILE_H + T.row] = m;
}

// FAST path: an upper bound of the running z of n fragments (n <= 64) from
// z0 on.  z_k = fl(z_{k-1} + dz) never rises when dz <= 0, so its maximum is
// z0; for dz > 0 (all values positive, normal range) k <= 63 rounded
// additions stay within (1+2^-24)^k of z0 + k dz, and fl(z0 + k dz) is
// within (1-2^-24)^2 of it, so fl(e * (1 + 2^-16)) bounds every z_k.
// Otherwise NaN: no bound (comparisons with it are false, so nothing is
// skipped; a NaN z never passes Less either).
__device__ __forceinline__ float depth_bound(float z0, float dz, uint32_t n) {
    const float e = fmul(fadd(z0, fmul((float)(n - 1u), dz)), 1.0000152587890625f);  // 1 + 2^-16
    return dz <= 0.0f ? z0 : dz > 0.0f && z0 >= 1e-30f ? e : __int_as_float(0x7FFFFFFF);
}

// ... and true when no fragment a..b-1 of a span can pass Less: the bound is
// <= the current depth of every pixel it covers.
__device__ __forceinline__ bool span_hidden(const TileCtx &T, float za, float dz, uint32_t a, uint32_t b) {
    const uint32_t s0 = (a - T.tx0) / RF_SEG, s1 = (b - 1u - T.tx0) / RF_SEG;
    float lo = T.smin[s0 * RF_TILE_H + T.row];
    for (uint32_t s = s0 + 1; s <= s1; ++s) lo = fminf(lo, T.smin[s * RF_TILE_H + T.row]);
    return depth_bound(za, dz, b - a) <= lo;
}

// rfx::jump out of line: the rasteriser's loop has to stay small (its
// instructions are fetched again on every pass).
static __device__ __noinline__ float jump_far(float s, float d, uint32_t k) { return jump(s, d, k); }

// The lane's scanline j of half H (raster.rs:84-113), clipped to the tile,
// then its fragments (raster.rs:60-69) into the tile (target.rs:163-198).
// FAST: the default context (depth test Less, colour and depth writes on).
// rv: the row's quantities, where the lane walks them.
template <int KIND, bool FAST>
__device__ __forceinline__ void span(TileCtx &T, const Paint &d, const HalfRec *__restrict__ H,
                                     const HalfRuns *__restrict__ U, uint32_t j, bool walked, const float *rv) {
    constexpr int NC = Kind<KIND>::NC;
    const float lx = walked ? rv[RF_R_LX] : row_value(H, U, RF_R_LX, j);
    const float rx = walked ? rv[RF_R_RX] : row_value(H, U, RF_R_RX, j);
    const float x0r = round_up_to_half(lx), x1r = round_up_to_half(rx);
    // xs..xe as `as usize` (target.rs:259-262), zip-truncated to the
    // fragment count, clipped to the tile.  32-bit saturating casts give the
    // same clipped range as 64-bit ones (tile columns are < 2^16), and keep
    // the conversions off the FP64 pipe.
    const uint32_t xs = as_u32(x0r);
    if (xs >= T.tx1) return;
    uint32_t xe = as_u32(x1r);
    if (xe < xs) xe = xs;
    uint32_t nfr = xe - xs;
    const uint32_t cnt = as_u32(fsub(x1r, x0r));
    if (cnt < nfr) nfr = cnt;
    const uint32_t a = xs > T.tx0 ? xs : T.tx0;
    const uint32_t b = nfr >= T.tx1 - xs ? T.tx1 : xs + nfr;
    if (a >= b) return;
    // v0 = left.next(); v0 = v0.lerp(v0.step(dv_dx), x0 - v0.x)  (raster.rs:88-102),
    // then k0 pixel steps to the tile's first column.
    const float tshift = fsub(x0r, lx);
    const uint32_t k0 = a - xs;
    float v[NC], dv[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        dv[c] = H->dvdx[c];
        const float c0 = walked ? rv[RF_R_C + c] : row_value(H, U, RF_R_C + c, j);
        const float adj = fadd(c0, fmul(fsub(fadd(c0, dv[c]), c0), tshift));
        v[c] = jump(adj, dv[c], k0);
    }
    constexpr int NP = PreNC<KIND>::NP;
    float2 v2[NP], dv2[NP];
#pragma unroll
    for (int c = 0; c < NP; ++c) {
        v2[c] = make_float2(v[2 * c], 2 * c + 1 < NC ? v[2 * c + 1 < NC ? 2 * c + 1 : 0] : 0.0f);
        dv2[c] = make_float2(dv[2 * c], 2 * c + 1 < NC ? dv[2 * c + 1 < NC ? 2 * c + 1 : 0] : 0.0f);
    }
    uint32_t idx = (a - T.tx0) * RF_TILE_H + T.row;
    const uint32_t end = (b - T.tx0) * RF_TILE_H + T.row;
    constexpr int U_PX = FAST && !Kind<KIND>::TEXTURED ? 4 : 1;
    while (idx < end) T.frags_o += px_group<KIND, FAST, U_PX>(T, d, (uint32_t)KIND, v2, dv2, idx, end);
}

// Which scanline of a half lands on row y: row(j) = (y0r + j) as usize =
// max(0, Y + j) with Y = y0r - 1/2.  Returns the j range [j0, j1) for row y
// (one scanline for rows below the top edge; row 0 also collects the rows
// above the buffer).
__device__ __forceinline__ void rows_for(const HalfRec *__restrict__ H, uint32_t y, uint32_t &j0,
                                         uint32_t &j1) {
    j0 = j1 = 0;
    const uint32_t n = H->n;
    const float y0r = H->y0r;
    if (n == 0 || !(fabsf(y0r) < RF_MAX_COORD)) return;
    const int32_t Y = (int32_t)fsub(y0r, 0.5f);
    if (y > 0 || Y >= 0) {
        const int64_t j = (int64_t)y - Y;
        if (j >= 0 && j < (int64_t)n) {
            j0 = (uint32_t)j;
            j1 = j0 + 1;
        }
    } else {
        j1 = (uint32_t)min((int64_t)n, (int64_t)1 - Y);
    }
}

template <int KIND, bool FAST>
__device__ __forceinline__ void raster_prim_k(TileCtx &T, const Paint &d, const PrimRec *__restrict__ P) {
    if (!T.row_ok) return;
    // The two halves cover disjoint rows, so each lane walks only the half
    // holding its row and both halves run in one pass of the warp.  Only
    // row 0 can take scanlines of both halves (rows above the buffer).
    uint32_t a0, a1, b0, b1;
    rows_for(&P->half[0], T.y, a0, a1);
    rows_for(&P->half[1], T.y, b0, b1);
    const bool start1 = a1 == a0;
    const HalfRec *H = start1 ? &P->half[1] : &P->half[0];
    const HalfRuns *U = start1 ? &P->runs[1] : &P->runs[0];
    uint32_t j = start1 ? b0 : a0, jend = start1 ? b1 : a1;
    bool more = !start1 && b1 > b0;
    // The rows above the buffer, all of them one lane's, are walked
    // (ScanlineIter::next); a single row's quantities are worked out as asked.
    constexpr int NQ = RF_R_C + Kind<KIND>::NC;
    float rv[NQ];
    bool walked = false;
    for (;;) {
        if (j >= jend) {
            if (!more) break;
            H = &P->half[1];
            U = &P->runs[1];
            j = b0;
            jend = b1;
            more = false;
            walked = false;
            continue;
        }
        if (!walked && jend - j > 1u) {
            walked = true;
#pragma unroll
            for (int r = 0; r < NQ; ++r) rv[r] = row_value(H, U, r, j);
        }
        span<KIND, FAST>(T, d, H, U, j, walked, rv);
        ++j;
        if (walked) {
#pragma unroll
            for (int r = 0; r < NQ; ++r) rv[r] = fadd(rv[r], H->d[r]);
        }
    }
}

// Row records in shared memory: one slot of row_words(NC) words per lane,
// word w of lane L at w * 32 + L (the bank is the lane).
// The row record at src into this lane's part of a slot (cp.async, 4 bytes a
// word), or an empty span (word 0 = 0) for a lane without one.
template <int KIND>
__device__ __forceinline__ void stage_row(uint32_t *slot, uint32_t lane, bool present, uint32_t kind,
                                          const uint32_t *src) {
    uint32_t *dst = slot + lane;
    if (!present) {
        dst[0] = 0u;
        return;
    }
    const uint32_t nw = KIND == RF_K_ANY ? row_words((int)kind_nc(kind)) : row_words(PreNC<KIND>::NC);
#pragma unroll
    for (uint32_t w = 0; w < row_words(PreNC<KIND>::NC); ++w) {
        if (w < nw) {
            const uint32_t sa = (uint32_t)__cvta_generic_to_shared(dst + w * RF_TILE_H);
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sa), "l"(src + w) : "memory");
        }
    }
}

// One item -- a scanline of a triangle inside the tile: its record sits in
// this lane's part of a slot (rs), its span [a, b) is clipped to the tile
// (xs: the span's first pixel).  v, dv: its varyings at pixel a and their
// steps.  A span that starts left of the tile takes the steps between: up to
// RF_STEP_MAX of them one after the other (two components an instruction: 64
// instructions for 32 pixels of Gouraud, where the exact jump takes about 100
// a component), more by the jump, in place.  (Records that also held the
// varyings at the first tile boundary saved up to a tile's steps here, but
// were nearly twice as long.)  The line at 128 steps, where lanes that jump no
// longer wait for each other's branches, was too low by the slowest tile: a
// round of jumps takes 5,000 cycles, 512 steps 2,000 (raster of a cube 300 px
// wide 26 -> 19 us, of 10,000 objects 116 -> 101; 256, 1,024 and 4,096 measure
// the same).
#define RF_STEP_MAX 512u
template <int KIND>
__device__ __forceinline__ void item_load(const float *dvdx, uint32_t *rs, uint32_t nc, uint32_t k, float2 *v,
                                          float2 *dv) {
    constexpr int NC = PreNC<KIND>::NC, NP = PreNC<KIND>::NP;
    if (k > RF_STEP_MAX) {
#pragma unroll 1
        for (uint32_t c = 0; c < nc; ++c)
            rs[(1u + c) * RF_TILE_H] = f2u(jump_far(u2f(rs[(1u + c) * RF_TILE_H]), dvdx[c], k));
        k = 0;
    }
#pragma unroll
    for (int c = 0; c < NP; ++c) {
        dv[c] = reinterpret_cast<const float2 *>(dvdx)[c];
        v[c].x = u2f(rs[(1 + 2 * c) * RF_TILE_H]);
        v[c].y = 2 * c + 1 < NC ? u2f(rs[(2 + 2 * c) * RF_TILE_H]) : 0.0f;
    }
#pragma unroll 1
    for (; k >= 4u; k -= 4u) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
#pragma unroll
            for (int c = 0; c < NP; ++c) v[c] = __fadd2_rn(v[c], dv[c]);
        }
    }
#pragma unroll
    for (uint32_t i = 0; i < 3; ++i)
        if (i < k) {
#pragma unroll
            for (int c = 0; c < NP; ++c) v[c] = __fadd2_rn(v[c], dv[c]);
        }
}

// A triangle without row records, from its PrimRec: lane = row (T.row = lane).
template <int KIND, bool FAST>
__device__ __noinline__ uint32_t raster_prim_slow(TileCtx T, uint32_t kind, const DrawDev *__restrict__ draw,
                                                  const PrimRec *__restrict__ P) {
    T.frags_o = 0;
    const Paint d(*draw);
    if constexpr (KIND != RF_K_ANY) {
        raster_prim_k<KIND == RF_K_ANY ? 0 : KIND, FAST>(T, d, P);
    } else {
        switch (kind) {
            case RF_K_FLAT: raster_prim_k<RF_K_FLAT, FAST>(T, d, P); break;
            case RF_K_GOURAUD: raster_prim_k<RF_K_GOURAUD, FAST>(T, d, P); break;
            case RF_K_TEXTURED: raster_prim_k<RF_K_TEXTURED, FAST>(T, d, P); break;
            case RF_K_TEX_GOURAUD: raster_prim_k<RF_K_TEX_GOURAUD, FAST>(T, d, P); break;
            default: raster_prim_k<RF_K_GOURAUD_SRGB, FAST>(T, d, P); break;
        }
    }
    return (uint32_t)T.frags_o;
}

// FAST path: the least current depth over the tile's rows this warp owns
// (a lower bound: the segment minima are), warp-uniform.
template <int TW>
__device__ __forceinline__ float tile_depth_min(const TileCtx &T) {
    float m = __int_as_float(0x7F800000);
    if (T.row_ok)
        for (uint32_t sg = 0; sg < (uint32_t)TW / RF_SEG; ++sg) m = fminf(m, T.smin[sg * RF_TILE_H + T.row]);
#pragma unroll
    for (int sft = 16; sft > 0; sft >>= 1) m = fminf(m, __shfl_xor_sync(0xFFFFFFFFu, m, sft));
    return m;
}

// Warp-wide selection of set bits in order: lane L offers the bits b (lane
// order, then bit order within a word); the first `want` of them go to the
// output slots first, first + 1, ...  Lane first + k learns where its bit
// came from (src lane, bit pos).  take = how many were handed out, total =
// how many were offered; end_lane / end_rest: the lane of the last bit taken
// and its bits still left.
struct WarpTake {
    uint32_t take, total, src, pos, end_lane, end_rest;
};
// (Out of line: it runs once per 32 triangles, and the kernels that switch
// on the shader kind per triangle are large already.)
static __device__ __noinline__ WarpTake warp_take(uint32_t b, uint32_t want, uint32_t first, uint32_t lane) {
    WarpTake t;
    const uint32_t c = __popc(b);
    uint32_t incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= (uint32_t)o) incl += y;
    }
    t.total = __shfl_sync(0xFFFFFFFFu, incl, 31);
    t.take = min(want, t.total);
    // Slot k = lane - first comes from the first lane whose inclusive count
    // exceeds k.
    const uint32_t k = lane - first;  // huge for lane < first: ignored
    uint32_t L = 0;
#pragma unroll
    for (uint32_t step = 16; step >= 1; step >>= 1) {
        const uint32_t v = __shfl_sync(0xFFFFFFFFu, incl, L + step - 1);
        if (v <= k) L += step;
    }
    const uint32_t ex = incl - c;
    const uint32_t exL = __shfl_sync(0xFFFFFFFFu, ex, L);
    const uint32_t bL = __shfl_sync(0xFFFFFFFFu, b, L);
    t.src = L;
    t.pos = nth_bit(bL, k - exL + 1u);  // (meaningless on lanes outside the take)
    // Where the take stopped: the source of slot take - 1.
    const uint32_t last = first + (t.take ? t.take : 1u) - 1u;
    t.end_lane = __shfl_sync(0xFFFFFFFFu, L, last & 31u);
    const uint32_t end_ex = __shfl_sync(0xFFFFFFFFu, exL, last & 31u);
    const uint32_t end_b = __shfl_sync(0xFFFFFFFFu, bL, last & 31u);
    const uint32_t used = t.take - end_ex;  // bits of end_lane taken
    const uint32_t lastpos = nth_bit(end_b, used ? used : 1u);
    t.end_rest = used ? (end_b & ~((2u << lastpos) - 1u)) : end_b;
    return t;
}

// Walks a tile's bitmask in submission order: set bits of the mask words
// (input triangles), each expanded to its clipped output triangles.  The
// tile's summary words (one bit per nonzero mask word) are read 128 at a
// time; the nonzero mask words they name are then fetched 32 at a time
// (lane e loads entry e), so an empty stretch of the mask costs nothing.
// Both gathers pick their next 32 set bits with one warp-wide prefix count
// (warp_take), not bit by bit.  Warp-uniform state; every lane calls
// gather_tris() together.
struct PrimIter {
    const uint32_t *tmask;  // the tile's mask words
    const uint32_t *tsum;   // the tile's summary words
    uint32_t nsum, tri_base, lane;
    // Summary words, 128 at a time: lane L holds words sb + 32 c + L in
    // s[c]; the cursor is chunk sc, lane sl, and srem = the bits of that
    // lane's word not taken yet (words of lower lanes are taken).
    uint32_t sb, s0, s1, s2, s3, sc, sl, srem;
    // Gathered mask words: lane e holds entry e (index widx, value wval),
    // wn of them; the cursor is entry wi with wrem = its bits not taken yet.
    uint32_t widx, wval, wn, wi, wrem;
    uint32_t fidx, fval, fn;  // the word batch after it
    bool started, done;           // a window was loaded; the summary words are all read

    __device__ __forceinline__ uint32_t chunk_word() const {
        return sc == 0 ? s0 : (sc == 1 ? s1 : (sc == 2 ? s2 : s3));
    }
    // The batch fetched ahead becomes the word batch, and the next up to 32
    // nonzero mask words, in order, are fetched.
    __device__ __forceinline__ void gather_words() {
        wn = fn;
        widx = fidx;
        wval = fval;
        wi = 0;
        wrem = __shfl_sync(0xFFFFFFFFu, wval, 0);
        fetch_words();
    }
    __device__ __forceinline__ void fetch_words() {
        uint32_t n = 0, mine = 0;
        while (!done) {
            if (!started || sc == 4) {  // next window of summary words
                if (started) sb += 128;
                started = true;
                if (sb >= nsum) {
                    done = true;
                    break;
                }
                const uint32_t i0 = sb + lane;
                s0 = i0 < nsum ? tsum[i0] : 0u;
                s1 = i0 + 32 < nsum ? tsum[i0 + 32] : 0u;
                s2 = i0 + 64 < nsum ? tsum[i0 + 64] : 0u;
                s3 = i0 + 96 < nsum ? tsum[i0 + 96] : 0u;
                sc = 0;
                sl = 0;
                srem = __shfl_sync(0xFFFFFFFFu, s0, 0);
            }
            const uint32_t w = chunk_word();
            const uint32_t b = lane < sl ? 0u : (lane == sl ? srem : w);
            if (__ballot_sync(0xFFFFFFFFu, b != 0u) == 0u) {  // nothing left in this chunk
                if (++sc < 4) {
                    sl = 0;
                    srem = __shfl_sync(0xFFFFFFFFu, chunk_word(), 0);
                }
                continue;
            }
            WarpTake t = warp_take(b, 32u - n, n, lane);
            if (lane >= n && lane < n + t.take) mine = (sb + sc * 32u + t.src) * 32u + t.pos;
            n += t.take;
            if (t.take < t.total) {  // stopped inside this chunk
                sl = t.end_lane;
                srem = t.end_rest;
                break;
            }
            ++sc;  // chunk used up
            if (sc < 4) {
                sl = 0;
                srem = __shfl_sync(0xFFFFFFFFu, chunk_word(), 0);
            }
            if (n == 32u) break;
        }
        fn = n;
        fidx = mine;
        fval = lane < n ? tmask[mine] : 0u;
    }
    // The next up to 32 input triangles (set bits), in order: lane k holds
    // the k-th one's global index in mine; returns how many.
    __device__ __forceinline__ uint32_t gather_tris(uint32_t &mine) {
        uint32_t n = 0;
        mine = 0;
        while (n < 32u) {
            if (wi >= wn) {
                if (fn == 0u) break;  // no mask words left
                gather_words();
            }
            const uint32_t b = (lane < wi || lane >= wn) ? 0u : (lane == wi ? wrem : wval);
            WarpTake t = warp_take(b, 32u - n, n, lane);
            const uint32_t wsrc = __shfl_sync(0xFFFFFFFFu, widx, t.src);
            if (lane >= n && lane < n + t.take) mine = tri_base + wsrc * 32u + t.pos;
            n += t.take;
            if (t.take < t.total) {  // stopped inside this word batch
                wi = t.end_lane;
                wrem = t.end_rest;
            } else {
                wi = wn;  // batch used up
            }
        }
        return n;
    }
    // From summary word `first` on (to nsum).
    __device__ __forceinline__ void init(uint32_t first) {
        sb = first;
        s0 = s1 = s2 = s3 = sc = sl = srem = 0;
        widx = wval = wn = wi = wrem = 0;
        started = done = false;
        fn = 0;
        fetch_words();
    }
};

// The next up to 32 entries of a list piece that did not fit, from the tile's
// masks (0 with y = 0 for none), n of them.  (Out of line, the iterator in
// local memory: a frame or two until the library has grown the lists.)
static __device__ __noinline__ uint2 mask_batch(PrimIter *it, const uint2 *ent, uint32_t lane, uint32_t *n) {
    uint32_t mine;
    const uint32_t k = it->gather_tris(mine);
    *n = k;
    return lane < k ? ent[mine] : make_uint2(0u, 0u);
}
static __device__ __noinline__ void mask_begin(PrimIter *it, const uint32_t *mask, const JobDev *J, uint32_t lt,
                                               uint32_t piece, uint32_t lane) {
    it->tmask = mask + J->mask_base + (size_t)lt * J->mask_words;
    it->tsum = mask + J->sum_base + (size_t)lt * J->sum_words;
    it->nsum = min((piece + 1u) * J->seg_words, J->sum_words);
    it->tri_base = J->tri_base;
    it->lane = lane;
    it->init(piece * J->seg_words);
}

// One commit group per call on every lane (copies issued since the last).
__device__ __forceinline__ void commit_stage() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }

// All but the N most recent groups of this lane complete, and visible to
// the whole warp.
template <int N>
__device__ __forceinline__ void wait_staged_but() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
    __syncwarp();
}

}  // namespace rfr

// Shared-memory words per warp: the colour and depth tiles, a work region,
// the depth-segment minima.  The work region is the row-major staging of the
// coalesced tile load and store (32 rows of min(TW, 32) + 1 words) while a
// tile moves, and between the two, in this order: the ring of output
// triangles not looked at yet, the table of the triangles being drawn (a
// uint4, the pixel steps, the draw and the depth bound of each), each row's
// current table entry, the queue of segments, two slots of row records.
constexpr uint32_t RF_CAND_WORDS = 256u;  // 31 left over and a batch of 32 fans fit
static_assert(31 + 32 * RF_MAX_FAN <= RF_CAND_WORDS, "ring size");
constexpr uint32_t RF_TAB_WORDS = (4u + 2u * RF_NC + 2u) * 32u;
// By row from this many scanlines a triangle in the tile: at 6 the grid's
// raster takes 107 us and the crates' 63, at 10 and at 16 84 and 51 (width 8);
// 64 uneven scenes 530 at 6 and 10, 545 at 16; the fill frame's triangles (18
// rows) are even at all three.
constexpr uint32_t RF_ROW_MEAN = 10u;
template <int TW, int KIND>
struct Region {
    static constexpr int NC = rfr::PreNC<KIND>::NC, NP = rfr::PreNC<KIND>::NP;
    static constexpr uint32_t QN = RF_TILE_H * ((uint32_t)TW / RF_SEG);  // segments of a tile
    static constexpr uint32_t QUEUE = QN * (1u + NC);
    static constexpr uint32_t SLOT = rfr::row_words(NC) * RF_TILE_H;
    static constexpr uint32_t WORDS = RF_CAND_WORDS + RF_TAB_WORDS + RF_TILE_H + QUEUE + 2u * SLOT;
};
template <int TW>
__host__ __device__ constexpr uint32_t raster_stage_words() {
    return RF_TILE_H * ((TW < 32 ? (uint32_t)TW : 32u) + 1u);
}
template <int TW, int KIND>
__host__ __device__ constexpr uint32_t raster_warp_words() {
    return 2u * TW * RF_TILE_H +
           (Region<TW, KIND>::WORDS > raster_stage_words<TW>() ? Region<TW, KIND>::WORDS : raster_stage_words<TW>()) +
           ((uint32_t)TW / RF_SEG) * RF_TILE_H;
}

namespace rfr {

// Coalesced transfer between a tile's global rows and its column-major
// shared-memory copy (word x * 32 + r): 16-byte accesses with the lanes of a
// row side by side (8 lanes per 128 bytes), through a row-major staging
// buffer of stride CB + 1 (CB = columns per pass, at most 32) whose odd
// stride keeps both sides free of bank conflicts.  Only the rows with bit r
// of `want` set are moved.  Every moved row must hold TW columns inside the
// target and start 16-byte aligned.
template <int TW, bool LOAD>
__device__ __forceinline__ void tile_rows_coalesced(uint32_t *__restrict__ tile, uint32_t *__restrict__ stg,
                                                    uint32_t *__restrict__ g, uint32_t pitch,
                                                    uint32_t want, uint32_t lane) {
    constexpr uint32_t CB = TW < 32 ? TW : 32;   // columns per pass
    constexpr uint32_t LPR = CB / 4;             // lanes per row
    constexpr uint32_t RPI = 32 / LPR;           // rows per instruction
    constexpr uint32_t SS = CB + 1;              // staging stride
    const uint32_t lr = lane / LPR, lc = (lane % LPR) * 4;
#pragma unroll 1
    for (uint32_t x0 = 0; x0 < (uint32_t)TW; x0 += CB) {
        if constexpr (LOAD) {
#pragma unroll
            for (uint32_t r0 = 0; r0 < 32; r0 += RPI) {
                const uint32_t r = r0 + lr;
                if ((want >> r) & 1u) {
                    const uint4 v = *reinterpret_cast<const uint4 *>(g + (size_t)r * pitch + x0 + lc);
                    uint32_t *d = stg + r * SS + lc;
                    d[0] = v.x;
                    d[1] = v.y;
                    d[2] = v.z;
                    d[3] = v.w;
                }
            }
            __syncwarp();
#pragma unroll 4
            for (uint32_t x = 0; x < CB; ++x) tile[(x0 + x) * RF_TILE_H + lane] = stg[lane * SS + x];
            __syncwarp();
        } else {
#pragma unroll 4
            for (uint32_t x = 0; x < CB; ++x) stg[lane * SS + x] = tile[(x0 + x) * RF_TILE_H + lane];
            __syncwarp();
#pragma unroll
            for (uint32_t r0 = 0; r0 < 32; r0 += RPI) {
                const uint32_t r = r0 + lr;
                if ((want >> r) & 1u) {
                    const uint32_t *sp = stg + r * SS + lc;
                    *reinterpret_cast<uint4 *>(g + (size_t)r * pitch + x0 + lc) = make_uint4(sp[0], sp[1], sp[2], sp[3]);
                }
            }
            __syncwarp();
        }
    }
}

// The tile's write-back as bulk copies (cp.async.bulk, the copy engine's
// untiled form), for tiles of whole 32-column blocks whose rows start
// 16-byte aligned.  Each 32 x 32 block of the column-major colour tile,
// then of the depth tile, is transposed into 32 rows of exactly 128 bytes
// -- lane r writes word x of row r at step k = x - r (mod 32), so both the
// column reads and the row writes hit 32 different banks -- and lane r
// hands row r to the copy engine as one 128-byte copy.  The first block
// goes to the staging area, every later one into the block read just
// before it (free once read), so no copy is waited for here: the caller
// waits (bulk_store_drain) before it next writes the tile or the staging
// area.  Rows without bit r of `want` are not copied.
template <int TW>
__device__ __forceinline__ void tile_store_bulk(uint32_t *__restrict__ scol, uint32_t *__restrict__ sdep,
                                                bool has_depth, uint32_t *__restrict__ stg,
                                                uint32_t *__restrict__ gcol, uint32_t *__restrict__ gdep,
                                                uint32_t pitch, uint32_t want, uint32_t lane) {
    static_assert(TW % 32 == 0, "whole 32-column blocks");
    constexpr uint32_t NB = (uint32_t)TW / 32u, BW = 32u * RF_TILE_H;  // blocks per buffer, words per block
    uint32_t *dst = stg;
#pragma unroll 1
    for (uint32_t m = 0; m < (has_depth ? 2u * NB : NB); ++m) {
        const uint32_t bi = m < NB ? m : m - NB;  // block within its buffer
        uint32_t *src = (m < NB ? scol : sdep) + bi * BW;
        uint32_t *g = (m < NB ? gcol : gdep) + bi * 32u;
#pragma unroll 8
        for (uint32_t k = 0; k < 32; ++k) {
            const uint32_t x = (lane + k) & 31u;
            dst[lane * 32 + x] = src[x * RF_TILE_H + lane];
        }
        // (rows written through the generic path, read by the copy engine)
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        __syncwarp();
        if ((want >> lane) & 1u) {
            const uint32_t sa = (uint32_t)__cvta_generic_to_shared(dst + lane * 32);
            asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], 128;\n" ::"l"(
                             g + (size_t)lane * pitch),
                         "r"(sa)
                         : "memory");
        }
        dst = src;
    }
    asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
}

// Every bulk copy this lane issued has read its shared-memory source (the
// tile and the staging area may be written again once the warp is past it).
__device__ __forceinline__ void bulk_store_drain() {
    asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");
    __syncwarp();
}

}  // namespace rfr

struct RasterArgs {
    const JobDev *jobs;
    const DrawDev *draws;
    const PrimRec *prims;
    const RasterPrim *rprims;
    const uint32_t *rows;
    const uint2 *ent;  // the triangles' list entries
    const uint32_t *mask;
    const uint2 *segs, *list;  // the tiles' triangle lists
    const uint32_t *items, *first, *nfirst;  // the group's part of the work list
    uint32_t *queue;
    StatsDev *stats;
    uint32_t nj, ntiles;  // ntiles: the group's
};

namespace rfr {

// The rows [l, e) of a half (its first at row y, n of them) that can meet the
// columns [x0, x1), or a few more: its edges as lines, moved apart by a pixel
// and by what n rounded additions may be off (each at most half a unit in the
// last place of the largest; taken fourfold), and the row where each crosses
// the columns' border moved out by a row.
__device__ __forceinline__ void trim_rows(const HalfRec &H, uint32_t y, uint32_t n, uint32_t x0, uint32_t x1,
                                          uint32_t &l, uint32_t &e) {
    const float L = u2f(H.b0[RF_R_LX]), R = u2f(H.b0[RF_R_RX]), dl = H.d[RF_R_LX], dr = H.d[RF_R_RX];
    const float m = fmaxf(fmaxf(fabsf(L), fabsf(R)), fmaxf(fabsf(L + (float)n * dl), fabsf(R + (float)n * dr)));
    if (!(m < 1e7f && fabsf(dl) < 1e7f && fabsf(dr) < 1e7f)) return;
    const float off = 1.0f + (float)n * m * 2.4e-7f;
    // rows k with a + k d < 0
    auto below = [&](float a, float d) {
        const float t = fminf(fmaxf(__fdividef(-a, d), 0.0f), 1e6f);
        if (d > 0.0f) e = min(e, y + (uint32_t)t + 2u);
        else if (d < 0.0f) l = max(l, y + max((uint32_t)t, 1u) - 1u);
        else if (a >= 0.0f) e = l;
    };
    below(L - off - (float)x1, dl);
    below((float)x0 - R - off, -dr);
}

// One work item (a tile, or the row slice `slice` >= 1 of one) of job J.
// KIND: the shader kind of every draw of the job, or RF_K_ANY; FAST: the
// default context (depth test Less, colour and depth writes) on a target
// with depth.
template <int TW, int KIND, bool FAST>
__device__ __forceinline__ void raster_tile(const RasterArgs &A, const JobDev &J, uint32_t ji, uint32_t tile,
                                            uint32_t slice, uint32_t *smem, uint32_t lane) {
    constexpr uint32_t NONE = 0xFFFFFFFFu, FULL = 0xFFFFFFFFu;
    using G = Region<TW, KIND>;
    constexpr int NC = G::NC, NP = G::NP;
    constexpr uint32_t WORDS = raster_warp_words<TW, KIND>();
    uint32_t *scol = smem;
    float *sdep = reinterpret_cast<float *>(scol + TW * RF_TILE_H);
    uint32_t *stg = scol + 2 * TW * RF_TILE_H;  // the work region
    uint32_t *cand = stg;
    uint4 *tab = reinterpret_cast<uint4 *>(stg + RF_CAND_WORDS);
    float *tab_dv = reinterpret_cast<float *>(tab + 32);  // [entry][half][component]
    uint32_t *tab_draw = reinterpret_cast<uint32_t *>(tab_dv + 2u * RF_NC * 32u);
    float *tab_z = reinterpret_cast<float *>(tab_draw + 32);
    uint32_t *row_entry = tab_draw + 64;  // entry | half << 5 | kind << 8
    uint32_t *segq = row_entry + RF_TILE_H;
    uint32_t *rslots = segq + G::QUEUE;
    const uint32_t lt = tile - J.tile_base;
    const uint32_t tyi = lt / J.tiles_x, txi = lt - tyi * J.tiles_x;
    TileCtx T;
    T.scol = scol;
    T.sdep = sdep;
    T.smin = reinterpret_cast<float *>(scol + WORDS - ((uint32_t)TW / RF_SEG) * RF_TILE_H);
    T.row = lane;
    T.tx0 = txi * TW;
    T.tx1 = min(T.tx0 + (uint32_t)TW, J.w);
    const uint32_t ty0 = tyi * RF_TILE_H;
    T.y = ty0 + lane;
    constexpr uint32_t SLICE_H = RF_TILE_H / RF_SPLIT_K;
    T.row_ok = T.y < J.h && (slice == 0 || lane / SLICE_H == slice - 1u);
    T.has_depth = J.depth != nullptr;
    T.depth_test = J.depth_test;
    T.color_write = J.color_write != 0;
    T.keep_depth = T.has_depth && J.depth_write != 0;
    T.no_test = !T.has_depth || J.depth_test == RF_K_DEPTH_NONE;
    T.fmt = pack_selector(J.pixfmt);
    T.rfmt = rgb_selector(T.fmt);
    T.frags_o = 0;
    const uint32_t ncols = T.tx1 - T.tx0;
    const size_t row_off = (size_t)T.y * J.w + T.tx0;
    const uint32_t rows_ok = __ballot_sync(FULL, T.row_ok);
    // Coalesced 16-byte row transfers (tile_rows_coalesced) when the
    // tile's rows hold its full width and start 16-byte aligned.
    const bool vec = ((J.w | T.tx0) & 3u) == 0u && ncols == (uint32_t)TW &&
                     (((uintptr_t)J.color | (uintptr_t)J.depth) & 15u) == 0u;
    uint32_t *gcol = J.color + (size_t)ty0 * J.w + T.tx0;
    uint32_t *gdep = reinterpret_cast<uint32_t *>(J.depth) + (size_t)ty0 * J.w + T.tx0;
    auto load_tile = [&]() {
        const bool cc = J.clear_flags & 1u, cd = (J.clear_flags & 2u) != 0u;
        if (vec) {
            if (cc) {
                for (uint32_t x = 0; x < (uint32_t)TW; ++x) scol[x * RF_TILE_H + lane] = J.clear_px;
            } else {
                tile_rows_coalesced<TW, true>(scol, stg, gcol, J.w, rows_ok, lane);
            }
            if (T.has_depth) {
                if (cd) {
                    for (uint32_t x = 0; x < (uint32_t)TW; ++x) sdep[x * RF_TILE_H + lane] = J.clear_z;
                } else {
                    tile_rows_coalesced<TW, true>(reinterpret_cast<uint32_t *>(sdep), stg, gdep, J.w, rows_ok, lane);
                }
            }
        } else {
            for (uint32_t x = 0; x < (uint32_t)TW; ++x) {
                const uint32_t i = x * RF_TILE_H + lane;
                const bool in = T.row_ok && x < ncols;
                scol[i] = cc ? J.clear_px : (in ? J.color[row_off + x] : 0u);
                if (T.has_depth) sdep[i] = cd ? J.clear_z : (in ? J.depth[row_off + x] : 0.0f);
            }
        }
    };
    // FAST: the tile's least current depth (a lower bound of every pixel
    // a span may write), for skipping whole triangles (RasterPrim::zmax).
    // Columns past the target's edge hold +inf, so they bound nothing
    // (they are never written back).
    float tzmin = 0.0f;
    // The target rows of this item: the tile's, or its slice's.
    const uint32_t ys = slice ? ty0 + (slice - 1u) * SLICE_H : ty0;
    const uint32_t ye = min(slice ? ys + SLICE_H : ty0 + RF_TILE_H, J.h);
    const uint32_t below = (1u << lane) - 1u, upto = below | (1u << lane);
    // Pixels a lane has in flight: as many as the registers and the instruction
    // cache bear.  Texture with colour: 2 where 4 took 113 us instead of 99 on
    // 10,000 objects; a texture alone, packed: 8 where 2 took 53 instead of 51 on
    // 1,600 crates.
    constexpr int U_SEG = KIND == RF_K_ANY ? 1
                          : KIND == RF_K_GOURAUD_SRGB || KIND == RF_K_TEX_GOURAUD || !FAST ? 2 : 4;
    constexpr int U_PACK = KIND == RF_K_ANY ? 1 : KIND == RF_K_TEXTURED && FAST ? 8 : 2;
    // Two lanes a segment where a round leaves room: pays where a pixel costs a
    // texel or the general tests (rasters of 10,000 textured objects 113.7 ->
    // 108.8 us, of 20,000 sorted triangles without depth 117.2 -> 109.8), not
    // for Gouraud's (100,000 triangles 173.1 -> 178.2).
    constexpr bool PAIRS = !FAST || KIND == RF_K_TEXTURED || KIND == RF_K_TEX_GOURAUD;
    // Four lanes a span where a packed round has few (most of the 32 are hidden
    // ones): the crates' raster 55 -> 53 us.  Not for texture with colour (the
    // 10,000 objects 81 -> 76, but the 500 k-triangle grid, whose rounds are
    // full, 91 -> 94) nor Gouraud (64 scenes 512 -> 521).
    constexpr bool SPLIT = KIND == RF_K_TEXTURED || KIND == RF_K_GOURAUD_SRGB;
    // A tall triangle's rows that miss the tile's columns left out before their
    // records are read, by its edges (trim_rows): 38 of 100 records read were
    // such rows.  Raster of 7,000 triangles 44.5 -> 41.6 us, of 100,000 167.8 ->
    // 163.6, of 20,000 without depth 110.2 -> 101.8.  Not for triangles of 32
    // rows or fewer (64 scenes 511 -> 520 with those of 17 too, 516 without; 7,000
    // triangles 41.3) nor textured kinds (10,000 objects 81 -> 86).
    constexpr bool TRIM = KIND == RF_K_FLAT || KIND == RF_K_GOURAUD || KIND == RF_K_GOURAUD_SRGB;
    constexpr bool PAINTED = KIND != RF_K_GOURAUD && KIND != RF_K_GOURAUD_SRGB;  // shading reads the draw

    // The item at row `row` of table entry ki whose record is in this lane's
    // part rs of a slot: its span [a, b) in the tile, and the varyings it
    // starts with.  False when it has no pixels here.
    auto enter = [&](uint32_t ki, uint32_t row, uint32_t *rs, float2 *v, float2 *dv, uint32_t &a, uint32_t &b,
                     uint32_t &half, uint32_t &kind) -> bool {
        const uint32_t w0 = rs[0];
        const uint32_t xs = w0 & 0xFFFFu, xe = w0 >> 16;
        a = xs > T.tx0 ? xs : T.tx0;
        b = xe < T.tx1 ? xe : T.tx1;
        if (a >= b) return false;
        const uint4 e = tab[ki];
        if constexpr (KIND == RF_K_ANY) kind = e.z >> 16;
        half = row < ((e.z >> 8) & 0xFFu) ? 0u : 1u;
        const float *dvdx = tab_dv + (ki * 2u + half) * RF_NC;
        const uint32_t nc = KIND == RF_K_ANY ? kind_nc(kind) : (uint32_t)NC;
        item_load<KIND>(dvdx, rs, nc, a - xs, v, dv);
        return true;
    };
    // The record of row r of the entry's in-tile rows into this lane's part of a slot.
    auto stage = [&](uint32_t *slot, bool have, const uint4 &e, uint32_t r) {
        const uint32_t kd = e.z >> 16;
        const uint32_t stride = KIND == RF_K_ANY ? row_words((int)kind_nc(kd)) : row_words(NC);
        stage_row<KIND>(slot, lane, have, kd, A.rows + e.x + (size_t)r * stride);
        commit_stage();
    };

    // The tile's list, a batch of 32 entries at a time (the next one already
    // loaded: ent, n_ent of them): the entries the tile does not hide go on
    // to the ring as output triangles.
    bool walk = false;  // the piece's masks are walked (the list did not hold it)
    PrimIter it;
    const uint2 *segs = A.segs + J.seg_base + (size_t)lt * J.nseg;
    uint32_t sb = 0, slive = 0, ent_off = 0, ent_left = 0, n_ent = 0;
    uint2 seg = make_uint2(0u, 0u), ent = make_uint2(0u, 0u);
    auto next_entries = [&]() {
        n_ent = 0;
        while (ent_left == 0u) {
            if (walk) {
                ent = mask_batch(&it, A.ent, lane, &n_ent);
                if (n_ent) return;
                walk = false;
            }
            while (slive == 0u) {
                if (sb >= J.nseg) return;
                seg = sb + lane < J.nseg ? segs[sb + lane] : make_uint2(0u, 0u);
                slive = __ballot_sync(FULL, seg.y != 0u);
                sb += 32u;
            }
            const uint32_t k = __ffs(slive) - 1u;
            slive &= slive - 1u;
            ent_off = __shfl_sync(FULL, seg.x, k);
            ent_left = __shfl_sync(FULL, seg.y, k);
            if (ent_left == RF_SEG_WALK) {
                mask_begin(&it, A.mask, &J, lt, sb - 32u + k, lane);
                ent_left = 0u;
                walk = true;
            }
        }
        n_ent = min(ent_left, 32u);
        ent = lane < n_ent ? A.list[ent_off + lane] : make_uint2(0u, 0u);
        ent_off += n_ent;
        ent_left -= n_ent;
    };
    // `todo`: the lanes of the 32 output triangles taken whose triangle has
    // scanlines in the tile and is not on the table yet, `slows` those
    // without row records.
    uint32_t todo = 0, slows = 0;
    uint32_t rows0 = 0, full = 0;  // a triangle's rows in the tile before trimming, and the table's
    uint32_t p = NONE, nr = 0, a0hs = 0, rb = 0, hdraw = 0;
    float zmax = 0.0f;
    uint32_t chead = 0, ncand = 0;  // the ring
    uint32_t nt = 0;                // triangles on the table
    bool done = false;
    next_entries();
    const bool any = n_ent != 0u;
    const bool loaded = any || J.clear_flags != 0u;  // (the tile comes in to be drawn into or cleared)
    if (loaded) {
        load_tile();
        if constexpr (FAST) {
            for (uint32_t x = ncols; x < (uint32_t)TW; ++x) sdep[x * RF_TILE_H + lane] = __int_as_float(0x7F800000);
            for (uint32_t sg = 0; sg < (uint32_t)TW / RF_SEG; ++sg) seg_refresh(T, sg);
            tzmin = tile_depth_min<TW>(T);
        }
        __syncwarp();
    }
    while (any) {
        if (!todo && !done) {
            while (ncand < 32u && n_ent) {
                // FAST: a triangle whose depth bound is at most the tile's
                // least depth passes no fragment (the tile's depths only
                // rise; a NaN on either side never skips).
                const bool keep = lane < n_ent && !(FAST && __uint_as_float(ent.y) <= tzmin);
                const uint32_t q = ent.x & RF_ENT_MASK, fan = ent.x >> RF_ENT_SHIFT;  // outputs q .. q + fan
                const uint32_t km = __ballot_sync(FULL, keep);
                uint32_t at = chead + ncand + __popc(km & below);
                if (__any_sync(FULL, keep && fan)) {  // fans of clipped triangles among them
                    uint32_t more = keep ? fan : 0u;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const uint32_t y = __shfl_up_sync(FULL, more, o);
                        if (lane >= (uint32_t)o) more += y;
                    }
                    ncand += __shfl_sync(FULL, more, 31);
                    if (keep) {
                        at += more - fan;
                        for (uint32_t i = 1; i <= fan; ++i) cand[(at + i) & (RF_CAND_WORDS - 1u)] = q + i;
                    }
                }
                if (keep) cand[at & (RF_CAND_WORDS - 1u)] = q;
                ncand += __popc(km);
                next_entries();
            }
            __syncwarp();
            done = ncand == 0u;
            p = lane < ncand ? cand[(chead + lane) & (RF_CAND_WORDS - 1u)] : NONE;
            const uint32_t took = min(ncand, 32u);
            chead += took;
            ncand -= took;
            uint4 h0 = make_uint4(0u, 0u, 0u, 0u), h1 = h0, h2 = h0;
            if (p != NONE) {
                const uint4 *h = reinterpret_cast<const uint4 *>(A.rprims + p);
                h0 = __ldg(h);
                h1 = __ldg(h + 1);
                h2 = __ldg(h + 2);
            }
            nr = rows0 = 0;
            bool slow = false;
            if (p != NONE) {
                const bool live = (h0.y & RF_RP_LIVE) != 0u, recs = (h0.y & RF_RP_ROWS) != 0u;
                slow = live && !recs;
                zmax = __uint_as_float(h2.y);
                hdraw = h0.x;
                if (live && recs && !(FAST && zmax <= tzmin)) {
                    const uint32_t y0 = h1.y, c0 = h1.z, y1 = h1.w, c1 = h2.x;
                    uint32_t l0 = max(y0, ys), e0 = min(y0 + c0, ye);
                    uint32_t l1 = max(y1, ys), e1 = min(y1 + c1, ye);
                    if (TRIM && (h0.y & RF_RP_EDGES)) {
                        const uint32_t m0 = e0, m1 = l1;
                        rows0 = (c0 && l0 < e0 ? e0 - l0 : 0u) + (c1 && l1 < e1 ? e1 - l1 : 0u);
                        if (c0 && l0 < e0) trim_rows(A.prims[p].half[0], y0, c0, T.tx0, T.tx1, l0, e0);
                        if (c1 && l1 < e1) trim_rows(A.prims[p].half[1], y1, c1, T.tx0, T.tx1, l1, e1);
                        if (c0 && c1 && l0 < e0 && l1 < e1) {  // (the rows between, too: they stay one run)
                            e0 = m0;
                            l1 = m1;
                        }
                    }
                    const uint32_t n0 = c0 && l0 < e0 ? e0 - l0 : 0u, n1 = c1 && l1 < e1 ? e1 - l1 : 0u;
                    nr = n0 + n1;
                    rows0 = max(rows0, nr);  // (the halves meet: y1 = y0 + c0 where both have rows)
                    const uint32_t a0 = (n0 ? l0 : l1) - ty0;
                    a0hs = a0 | (a0 + n0) << 8 | h0.z << 16;
                    rb = h0.w + (n0 ? l0 - y0 : c0 + (l1 - y1)) * h1.x;
                }
            }
            slows = __ballot_sync(FULL, slow);
            todo = __ballot_sync(FULL, nr != 0u) | slows;
        }
        // Onto the table, up to the first triangle without records or until
        // it is full.
        {
            const uint32_t stop = slows & todo ? (uint32_t)__ffs(slows & todo) - 1u : 32u;
            const uint32_t m = stop < 32u ? todo & ((1u << stop) - 1u) : todo;
            const uint32_t at = nt + __popc(m & below);
            const bool put = ((m >> lane) & 1u) && at < 32u;
            if (put) {
                tab[at] = make_uint4(rb, nr, a0hs, p);
                tab_draw[at] = hdraw;
                tab_z[at] = zmax;
#pragma unroll
                for (uint32_t c = 0; c < 2u * RF_NC / 4u; ++c) {
                    const uint32_t sa = (uint32_t)__cvta_generic_to_shared(tab_dv + at * (2u * RF_NC) + 4u * c);
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(sa),
                                 "l"(&A.rprims[p].dvdx[0][0] + 4u * c)
                                 : "memory");
                }
            }
            const uint32_t took = __ballot_sync(FULL, put);
            nt += __popc(took);
            if (TRIM) full += __reduce_add_sync(FULL, put ? rows0 : 0u);
            todo &= ~took;
        }
        const uint32_t slow_now = todo && ((slows >> (__ffs(todo) - 1)) & 1u) ? todo & (0u - todo) : 0u;
        if (!todo && !done) continue;  // the table has room left

        // The table's triangles, scanline by scanline.  (Their steps arrive
        // with the first row records.)
        __syncwarp();
        if (nt) {
            const uint4 te = lane < nt ? tab[lane] : make_uint4(0u, 0u, 0u, 0u);
            const uint32_t n = te.y;
            uint32_t ex = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(FULL, ex, o);
                if (lane >= (uint32_t)o) ex += y;
            }
            const uint32_t total = __shfl_sync(FULL, ex, 31);
            ex -= n;
            float2 v[NP], dv[NP];
            uint32_t sl = 0;
            if ((TRIM ? full : total) >= RF_ROW_MEAN * nt) {
                // By row: lane r takes row r's triangles in order, one a
                // round, passing over those its row hides.  A round's spans
                // never meet; cut into segments of RF_SEG pixels, the
                // visible ones queue up and are drawn on full warps.
                uint32_t rm = n ? (n < 32u ? (1u << n) - 1u : FULL) << (te.z & 0xFFu) : 0u;  // this triangle's rows
#pragma unroll
                for (uint32_t sft = 16, m = 0x0000FFFFu; sft; sft >>= 1, m ^= m << sft) {
                    const uint32_t o = __shfl_xor_sync(FULL, rm, sft);
                    rm = lane & sft ? (rm & ~m) | ((o >> sft) & m) : (rm & m) | ((o << sft) & ~m);
                }  // now the triangles of this lane's row
                uint32_t kin = 0;
                bool haven = false;
                auto stage_next = [&]() {
                    haven = false;
                    if (rm) {
                        float rmin = -__int_as_float(0x7F800000);
                        if constexpr (FAST) {
                            rmin = T.smin[lane];
#pragma unroll
                            for (uint32_t sg = 1; sg < (uint32_t)TW / RF_SEG; ++sg)
                                rmin = fminf(rmin, T.smin[sg * RF_TILE_H + lane]);
                        }
                        do {  // the next one this row does not hide
                            kin = __ffs(rm) - 1u;
                            rm &= rm - 1u;
                            haven = !(FAST && tab_z[kin] <= rmin);
                        } while (!haven && rm);
                    }
                    const uint4 e = tab[kin];
                    stage(rslots + sl * G::SLOT, haven, e, lane - (e.z & 0xFFu));
                };
                stage_next();
                T.row = lane;
                while (__any_sync(FULL, haven)) {
                    const uint32_t ki = kin;
                    bool act = haven;
                    uint32_t *rs = rslots + sl * G::SLOT + lane;
                    sl ^= 1u;
                    stage_next();
                    wait_staged_but<1>();
                    uint32_t kind = (uint32_t)KIND, half = 0, a = 0, b = 0;
                    act = act && enter(ki, lane, rs, v, dv, a, b, half, kind);
                    uint32_t x = a - T.tx0;
                    const uint32_t xe = b - T.tx0;
                    if (act) row_entry[lane] = ki | half << 5 | kind << 8;
                    uint32_t nq = 0;
                    while (__any_sync(FULL, act)) {
                        const uint32_t sg = x / RF_SEG, xn = min(xe, (sg + 1u) * RF_SEG), len = xn - x;
                        bool vis = act;
                        if constexpr (FAST)
                            vis = act && !(depth_bound(v[0].x, dv[0].x, len) <= T.smin[sg * RF_TILE_H + lane]);
                        const uint32_t vm = __ballot_sync(FULL, vis);
                        if (vis) {
                            uint32_t *q = segq + nq + __popc(vm & below);
                            q[0] = (x * RF_TILE_H + lane) | len << 16;
#pragma unroll
                            for (int c = 0; c < NC; ++c) q[(1 + c) * G::QN] = f2u(c & 1 ? v[c / 2].y : v[c / 2].x);
                        }
                        nq += __popc(vm);
                        x = xn;
                        act = act && x < xe;
                        if (TW > (int)RF_SEG && act) {
#pragma unroll
                            for (uint32_t i = 0; i < RF_SEG; ++i)
                                if (i < len) {
#pragma unroll
                                    for (int c = 0; c < NP; ++c) v[c] = __fadd2_rn(v[c], dv[c]);
                                }
                        }
                    }
                    __syncwarp();
                    // (few: two lanes a segment, half of its pixels each)
                    const uint32_t pair = PAIRS && nq <= 16u ? 1u : 0u;
#pragma unroll 1
                    for (uint32_t j = lane; j < nq << pair; j += 32u) {
                        const uint32_t k = j >> pair, w = segq[k];
                        uint32_t idx = w & 0xFFFFu, end = idx + (w >> 16) * RF_TILE_H;
                        const uint32_t first = idx, row = idx & 31u;
                        const uint32_t re0 = row_entry[row], re = (re0 & 31u) * 2u + ((re0 >> 5) & 1u);
                        float2 sv[NP], sd[NP];
#pragma unroll
                        for (int c = 0; c < NP; ++c) {
                            sv[c].x = u2f(segq[k + (1 + 2 * c) * G::QN]);
                            sv[c].y = 2 * c + 1 < NC ? u2f(segq[k + (2 + 2 * c) * G::QN]) : 0.0f;
                            sd[c] = reinterpret_cast<const float2 *>(tab_dv + re * RF_NC)[c];
                        }
                        const Paint paint(A.draws[PAINTED ? tab_draw[re0 & 31u] : 0u]);
                        uint32_t nout = 0;
                        if (j & pair) {
                            idx += RF_SEG / 2u * RF_TILE_H;
#pragma unroll
                            for (uint32_t i = 0; i < RF_SEG / 2u; ++i)
#pragma unroll
                                for (int c = 0; c < NP; ++c) sv[c] = __fadd2_rn(sv[c], sd[c]);
                        } else if (pair) {
                            end = min(end, idx + RF_SEG / 2u * RF_TILE_H);
                        }
                        while (idx < end)
                            nout += px_group<KIND, FAST, U_SEG>(T, paint, KIND == RF_K_ANY ? re0 >> 8 : (uint32_t)KIND,
                                                                sv, sd, idx, end);
                        T.frags_o += nout;
                        if constexpr (FAST) {
                            // (both halves' depths before the segment's least)
                            if (pair) __syncwarp(nq == 16u ? FULL : (1u << 2u * nq) - 1u);
                            T.row = row;
                            if (nout) seg_refresh(T, first / (RF_SEG * RF_TILE_H));
                        }
                    }
                    __syncwarp();
                    T.row = lane;
                }
                // Where every row hides every triangle no round has waited for
                // the table's own copies; the next table, or the tile's
                // write-back, takes their place.
                wait_staged_but<0>();
            } else {
                // Packed: 32 scanlines a pass, in submission order, one a
                // lane.  Spans of one row that meet are drawn in that order:
                // each waits for the lower lanes it overlaps.
                if (n) tab[lane].y = ex;
                __syncwarp();
                uint32_t kin = 0, rown = 0;
                auto stage_pass = [&](uint32_t base) {
                    // the last triangle that starts at or before the item, and its row there
                    const uint32_t starts = __reduce_or_sync(FULL, n && ex - base < 32u ? 1u << (ex - base) : 0u);
                    const uint32_t before = __popc(__ballot_sync(FULL, n && ex < base));
                    const bool have = base + lane < total;
                    uint4 e = make_uint4(0u, 0u, 0u, 0u);
                    if (have) {
                        kin = before + __popc(starts & upto) - 1u;
                        e = tab[kin];
                        rown = (e.z & 0xFFu) + (base + lane - e.y);
                    }
                    stage(rslots + sl * G::SLOT, have, e, base + lane - e.y);
                };
                stage_pass(0u);
#pragma unroll 1
                for (uint32_t base = 0; base < total; base += 32u) {
                    uint32_t ki = kin, row = rown;
                    uint32_t *rs = rslots + sl * G::SLOT + lane;
                    sl ^= 1u;
                    stage_pass(base + 32u);
                    wait_staged_but<1>();
                    uint32_t kind = (uint32_t)KIND, half = 0, a = 0, b = 0;
                    T.row = row;
                    bool act = base + lane < total && enter(ki, row, rs, v, dv, a, b, half, kind);
                    if constexpr (FAST) act = act && !span_hidden(T, v[0].x, dv[0].x, a, b);
                    uint32_t pend = __ballot_sync(FULL, act);
                    uint32_t lower = __match_any_sync(FULL, act ? row : 32u + lane) & below;
                    uint32_t wait = 0;
                    while (__any_sync(FULL, lower != 0u)) {
                        const uint32_t src = lower ? (uint32_t)__ffs(lower) - 1u : lane;
                        const uint32_t oa = __shfl_sync(FULL, a, src), ob = __shfl_sync(FULL, b, src);
                        if (lower && oa < b && a < ob) wait |= 1u << src;
                        lower &= lower - 1u;
                    }
                    while (pend) {
                        bool go = ((pend >> lane) & 1u) && (wait & pend) == 0u;
                        const uint32_t gm = __ballot_sync(FULL, go), cnt = __popc(gm);
                        pend &= ~gm;
                        if (SPLIT && pend == 0u && cnt <= 8u) {
                            // The last ones, and few: four lanes a span.
                            const uint32_t src = nth_bit(gm, min(lane >> 2, cnt - 1u) + 1u);
                            go = lane >> 2 < cnt;
                            row = __shfl_sync(FULL, row, src);
                            ki = __shfl_sync(FULL, ki, src);
                            a = __shfl_sync(FULL, a, src);
                            b = __shfl_sync(FULL, b, src);
                            if (KIND == RF_K_ANY) kind = __shfl_sync(FULL, kind, src);
#pragma unroll
                            for (int c = 0; c < NP; ++c) {
                                v[c].x = __shfl_sync(FULL, v[c].x, src);
                                v[c].y = __shfl_sync(FULL, v[c].y, src);
                                dv[c].x = __shfl_sync(FULL, dv[c].x, src);
                                dv[c].y = __shfl_sync(FULL, dv[c].y, src);
                            }
                            const uint32_t part = (b - a + 3u) >> 2, skip = part * (lane & 3u);
#pragma unroll 1
                            for (uint32_t i = 0; i < skip; ++i) {
#pragma unroll
                                for (int c = 0; c < NP; ++c) v[c] = __fadd2_rn(v[c], dv[c]);
                            }
                            a += skip;
                            b = min(b, a + part);
                            go = go && a < b;
                            T.row = row;
                        }
                        uint32_t nout = 0;
                        if (go) {
                            const Paint paint(A.draws[PAINTED ? tab_draw[ki] : 0u]);
                            uint32_t idx = (a - T.tx0) * RF_TILE_H + row;
                            const uint32_t end = (b - T.tx0) * RF_TILE_H + row;
                            do nout += px_group<KIND, FAST, U_PACK>(T, paint, kind, v, dv, idx, end);
                            while (idx < end);
                            T.frags_o += nout;
                        }
                        if constexpr (FAST) {
                            if (SPLIT) __syncwarp();  // (all of a span's lanes' depths before the least)
                            if (nout)
                                for (uint32_t sg = (a - T.tx0) / RF_SEG; sg <= (b - 1u - T.tx0) / RF_SEG; ++sg)
                                    seg_refresh(T, sg);
                        }
                        __syncwarp();  // (the depths written before the next round reads them)
                    }
                }
                T.row = lane;
            }
            __syncwarp();
            nt = full = 0;
            if constexpr (FAST) tzmin = tile_depth_min<TW>(T);
        }
        if (slow_now) {
            const uint32_t l = __ffs(slow_now) - 1u;
            const uint32_t ps = __shfl_sync(FULL, p, l), ds = __shfl_sync(FULL, hdraw, l);
            T.frags_o += raster_prim_slow<KIND, FAST>(T, (uint32_t)A.draws[ds].shader, A.draws + ds, A.prims + ps);
            __syncwarp();
            todo &= ~slow_now;
        }
        if (done) break;
    }
    if (loaded) {
        if (vec) {
            if constexpr (TW % 32 == 0) {
                tile_store_bulk<TW>(scol, reinterpret_cast<uint32_t *>(sdep), T.has_depth, stg, gcol, gdep, J.w,
                                    rows_ok, lane);
            } else {
                tile_rows_coalesced<TW, false>(scol, stg, gcol, J.w, rows_ok, lane);
                if (T.has_depth)
                    tile_rows_coalesced<TW, false>(reinterpret_cast<uint32_t *>(sdep), stg, gdep, J.w, rows_ok, lane);
            }
        } else if (T.row_ok) {
            for (uint32_t x = 0; x < ncols; ++x) {
                const uint32_t i = x * RF_TILE_H + lane;
                J.color[row_off + x] = scol[i];
                if (T.has_depth) J.depth[row_off + x] = sdep[i];
            }
        }
    }
    __syncwarp();
    warp_add_u64(&A.stats[ji].frags_o, T.frags_o, true);
}

}  // namespace rfr

// Persistent warps over the work list of one raster group.
template <int TW, int KIND, bool FAST>
__global__ void __launch_bounds__(RF_RASTER_MAX_THREADS, 2) k_raster(const __grid_constant__ RasterArgs A) {
    using namespace rfr;
    grid_begin();
    extern __shared__ __align__(16) uint32_t smem[];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr uint32_t WARP_WORDS = raster_warp_words<TW, KIND>();
    static_assert(WARP_WORDS % 4u == 0u && (2u * TW * RF_TILE_H) % 4u == 0u,
                  "each warp's area and its staging start 16-byte aligned (bulk copies)");
    // Queue position q: the heavy tiles and crowded-tile slices first
    // (first[q]), then every other tile in index order.
    const uint32_t nfirst = *A.nfirst;
    const uint32_t nitems = A.ntiles + nfirst;
    for (;;) {
        uint32_t item = 0;
        if (lane == 0) {
            do {
                const uint32_t pos = atomicAdd(A.queue, 1u);
                item = pos >= nitems ? 0xFFFFFFFFu : (pos < nfirst ? A.first[pos] : A.items[pos - nfirst]);
            } while (item == RF_ITEM_SKIP);
        }
        item = __shfl_sync(0xFFFFFFFFu, item, 0);
        if (item == 0xFFFFFFFFu) break;
        const uint32_t tile = item >> RF_ITEM_SHIFT, slice = item & ((1u << RF_ITEM_SHIFT) - 1u);  // 0: the whole tile
        if constexpr (TW % 32 == 0) bulk_store_drain();  // (the last tile's write-back)
        const uint32_t ji = A.jobs[warp_find(A.nj, tile, [&](uint32_t i) { return A.jobs[i].nth_tile; })].nth;
        raster_tile<TW, KIND, FAST>(A, A.jobs[ji], ji, tile, slice, smem + warp * WARP_WORDS, lane);
    }
    // (shared memory stays allocated until the last write-back has read it)
    if constexpr (TW % 32 == 0) bulk_store_drain();
}

namespace rfk {

// The opt-in to more than 48 KB of dynamic shared memory is a property of
// each kernel on each device: set once per (kernel, device) -- the flags
// live in the instantiation for that kernel (Tag), since every k_raster
// variant has the same function type -- under a lock so host threads
// driving contexts on several devices may launch concurrently, and with
// its status returned.
template <class Tag, class K>
static cudaError_t opt_in_smem(K kernel, int bytes) {
    constexpr int MAX_DEV = 64;
    static std::mutex mu;
    static bool done[MAX_DEV] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= MAX_DEV) return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    std::lock_guard<std::mutex> lk(mu);
    if (!done[dev]) {
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (e != cudaSuccess) return e;
        done[dev] = true;
    }
    return cudaSuccess;
}

template <int TW, int KIND, bool FAST>
static cudaError_t launch_raster_k(RF_RASTER_PARAMS) {
    // Shared memory per block: at most the 227 KB opt-in limit, so the
    // block takes as many warps as fit (wide tiles of the generic kind).
    constexpr size_t SMEM_MAX = 227 * 1024;
    constexpr size_t per_warp = (size_t)raster_warp_words<TW, KIND>() * 4;
    if ((size_t)warps * per_warp > SMEM_MAX) warps = (uint32_t)(SMEM_MAX / per_warp);
    const size_t smem = (size_t)warps * per_warp;
    struct Tag {};  // one per (TW, KIND, FAST)
    cudaError_t e = opt_in_smem<Tag>(k_raster<TW, KIND, FAST>, (int)SMEM_MAX);
    if (e != cudaSuccess) return e;
    if (ntiles == 0) return cudaSuccess;  // (loaded)
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_raster<TW, KIND, FAST>, warps * 32, smem);
    if (per_sm < 1) per_sm = 1;
    uint32_t blocks = (uint32_t)per_sm * (uint32_t)nsm;
    const uint32_t need = (ntiles + warps - 1) / warps;  // (a few crowded-tile slices more are shared out)
    if (blocks > need) blocks = need;
    if (blocks == 0) blocks = 1;
    const RasterArgs A{jobs, draws, prims, rprims, rows, ent, mask, segs, list, items, first, nfirst, queue, stats, nj, ntiles};
    RF_NEXT(k_raster<TW, KIND, FAST>, blocks, warps * 32, smem, s, A);
    return cudaGetLastError();
}

// The launcher of one tile width and context: the kernel of the group's
// shader kind.
template <int TW, bool FAST>
static cudaError_t launch_raster_for_width(int kind, RF_RASTER_PARAMS) {
    switch (kind) {
        case RF_K_FLAT: return launch_raster_k<TW, RF_K_FLAT, FAST>(RF_RASTER_ARGS);
        case RF_K_GOURAUD: return launch_raster_k<TW, RF_K_GOURAUD, FAST>(RF_RASTER_ARGS);
        case RF_K_TEXTURED: return launch_raster_k<TW, RF_K_TEXTURED, FAST>(RF_RASTER_ARGS);
        case RF_K_TEX_GOURAUD: return launch_raster_k<TW, RF_K_TEX_GOURAUD, FAST>(RF_RASTER_ARGS);
        case RF_K_GOURAUD_SRGB: return launch_raster_k<TW, RF_K_GOURAUD_SRGB, FAST>(RF_RASTER_ARGS);
        default: return launch_raster_k<TW, RF_K_ANY, FAST>(RF_RASTER_ARGS);
    }
}

}  // namespace rfk

#endif
