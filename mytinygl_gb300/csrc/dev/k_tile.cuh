// k_tile.cuh — K4 tile raster/ROP (replaces rasterize_triangle_smooth's pixel loop,
// raster.c:532-724, and glClear's loops, gl_api.c:409-457).
//
// A CTA owns one tile (8, 16 or 32 pixels square); thread t owns one pixel for the whole pass,
// so the pixel's colour, depth and stencil stay in registers between fragments. Each warp
// covers an 8x4 block of the tile. Because a pixel is only ever touched by its own thread,
// in-order blending and stencil updates need no atomics. Clears of the pass are applied first;
// a clear that covers the whole tile means that buffer is never read from memory.
//
// k_tile (here) walks the tile's record list in submission order. Records are staged 32 or 64
// at a time into shared memory with asynchronous copies, the next chunk in flight while one is
// walked, so that the walk reads no global memory for them. Per chunk each lane tests a record
// or two against its warp's block (a corner test of the edges, the depth rejection), the lanes
// find which pixels each remaining record covers, as 32-bit masks, and the masks are transposed
// across the warp: every lane then holds the records of its own pixel, in order, and takes one
// per round through the reference's fragment pipeline: barycentrics, stencil test/ops, depth
// test, colour (flat / smooth / per-fragment lighting), texture with alpha test and texenv,
// fog, depth write, blend, masked write. Rounds are as many as the deepest pixel's records,
// whatever the records' sizes. Passes whose result does not depend on the order take k_tile_free.cu.
//
// What bounds it: issue of the fragment pipeline (blended sprites and small triangles).
#pragma once

#include <algorithm>

#include "dev_kernels.h"

namespace mtgl {

__device__ __forceinline__ bool covers_tile(const ClearOp &c, uint32_t bit, int x0, int y0, int x1, int y1)
{
    return (c.mask & bit) && c.x0 <= x0 && c.y0 <= y0 && c.x1 >= x1 && c.y1 >= y1;
}

// Float order as signed-int order (negative floats reversed), so a warp max is one REDUX.
__device__ __forceinline__ int ordered_key(float f)
{
    const int b = __float_as_int(f);
    return b ^ ((b >> 31) & 0x7FFFFFFF);
}
__device__ __forceinline__ float ordered_float(int k) { return __int_as_float(k ^ ((k >> 31) & 0x7FFFFFFF)); }

// Largest stored depth over the warp's pixels inside the framebuffer.
__device__ __forceinline__ float warp_max_depth(float dep, bool in_fb)
{
    return ordered_float(__reduce_max_sync(0xffffffffu, in_fb ? ordered_key(dep) : INT32_MIN));
}

constexpr uint32_t kNoPending = 0xFFFFFFFFu;

// ------------------------------------------------------------------ staging

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem)
{
    const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// 32x32 bit transpose across the warp: bit i of lane l becomes bit l of lane i (block swaps of
// halving size: Warren, "Hacker's Delight", 7-3, with lanes for words).
__device__ __forceinline__ uint32_t warp_transpose(uint32_t v)
{
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t mask = 0x0000FFFFu;
#pragma unroll
    for (int s = 16; s; s >>= 1) {
        // swap the off-diagonal s x s blocks of each 2s x 2s block with the lane s away
        const uint32_t o = __shfl_xor_sync(0xffffffffu, v, s);
        v = (lane & s) ? ((v & ~mask) | ((o & ~mask) >> s)) : ((v & mask) | ((o & mask) << s));
        mask ^= mask << (s >> 1);
    }
    return v;
}


// ------------------------------------------------------------------ tiles

// A warp's 8x4 block of a tile and its pixels' starting values.
struct TilePixel {
    int wx0, wy0, wx1, wy1;  // the block's part of the framebuffer (empty: wx1 < wx0 or wy1 < wy0)
    bool store_stencil;
    uint32_t col, st;
    float dep;
    __device__ int px() const { return wx0 + (int)(threadIdx.x & 7u); }
    __device__ int py() const { return wy0 + (int)((threadIdx.x >> 3) & 3u); }
    __device__ bool in_fb() const { return px() <= wx1 && py() <= wy1; }
};

// Loads the tile's buffers where no clear covers the tile, and applies the clears (those of the
// whole framebuffer come with the frame, which saves a dependent load per tile and their tests: 110 of
// an empty block's 369 instructions; 48 served requests 3.86 -> 3.64 ms). The stencil
// buffer is only touched when the pass may change it (`stencil`) or a clear does.
template <int TS>
__device__ __forceinline__ TilePixel open_tile(const TileArgs &A, const DevFrame &F, uint32_t tile, bool stencil)
{
    constexpr int kWarpsX = TS / 8;
    const int warp = threadIdx.x >> 5;
    const uint32_t local = tile - F.tile_base, row = tile_row(F, local);
    const int tx = (int)(local - row * (uint32_t)F.dims.tiles_x), ty = (int)row;
    const int W = F.dims.width, H = F.dims.height;
    TilePixel t;
    t.wx0 = tx * TS + (warp % kWarpsX) * 8;
    t.wy0 = ty * TS + (warp / kWarpsX) * 4;
    t.wx1 = min(t.wx0 + 7, W - 1);
    t.wy1 = min(t.wy0 + 3, H - 1);
    const int px = t.px(), py = t.py();
    uint32_t cleared = F.cleared;
    t.col = F.clear_color;
    t.dep = F.clear_depth;
    t.st = F.clear_stencil;
    bool load_c = !(cleared & GL_COLOR_BUFFER_BIT), load_d = !(cleared & GL_DEPTH_BUFFER_BIT);
    bool load_s = (stencil || F.host_stencil) && !(cleared & GL_STENCIL_BUFFER_BIT);
    const ClearOp *clears = A.clears + F.clear_base;
    const int nclears = (int)F.nclears;
    const int bx0 = tx * TS, by0 = ty * TS, bx1 = min(bx0 + TS, W), by1 = min(by0 + TS, H);
#pragma unroll 1
    for (int i = 0; i < nclears; i++) {
        const ClearOp &c = clears[i];
        cleared |= c.mask;
        if (covers_tile(c, GL_COLOR_BUFFER_BIT, bx0, by0, bx1, by1)) load_c = false;
        if (covers_tile(c, GL_DEPTH_BUFFER_BIT, bx0, by0, bx1, by1)) load_d = false;
        if (covers_tile(c, GL_STENCIL_BUFFER_BIT, bx0, by0, bx1, by1)) load_s = false;
        else if (c.mask & GL_STENCIL_BUFFER_BIT) load_s = true;
    }
    t.store_stencil = stencil || (cleared & GL_STENCIL_BUFFER_BIT) != 0;
    if (t.in_fb()) {
        const size_t pix = (size_t)py * W + px;
        if (load_c) t.col = F.color[pix];
        if (load_d) t.dep = F.depth[pix];
        if (load_s) t.st = F.stencil[pix];
#pragma unroll 1
        for (int i = 0; i < nclears; i++) {
            const ClearOp &c = clears[i];
            if (px >= c.x0 && px < c.x1 && py >= c.y0 && py < c.y1) {
                if (c.mask & GL_COLOR_BUFFER_BIT) t.col = c.color;
                if (c.mask & GL_DEPTH_BUFFER_BIT) t.dep = c.depth;
                if (c.mask & GL_STENCIL_BUFFER_BIT) t.st = c.stencil & 0xFFu;
            }
        }
    }
    return t;
}

// A tile's pixels on their way to the host.
template <int TS>
struct HostTile {
    uint32_t col[TS * TS];
    float dep[TS * TS];
    uint8_t st[TS * TS];
};

// Stores the tile, and what of it goes to page-locked host memory. With `rows` the latter go out in
// whole tile rows, through shared memory: the link takes 32-byte writes (a block's rows) at 144
// GB/s and 64-byte ones (a 16-pixel tile's rows) at 170. That is worth its instructions where a
// pixel is shaded once (order-free passes: phong 143 -> 130 us, textured 324 -> 310, 256 uneven
// frames 4.66 -> 4.57 ms, 48 served ones 3.64 -> 3.67) and not in ordered passes, which the
// fragments bound (4K sprites 965 -> 982 us, the million blended triangles the same).
template <int TS>
__device__ __forceinline__ void close_tile(const TileArgs &A, const DevFrame &F, const TilePixel &t, uint32_t col,
                                           float dep, uint32_t st, HostTile<TS> *rows)
{
    const int W = F.dims.width, H = F.dims.height;
    const size_t pix = (size_t)t.py() * W + t.px();
    if (t.in_fb()) {
        if (!debug_check(A.debug, pix < (size_t)W * (size_t)H, DBG_TILE_PIXEL)) return;
        F.color[pix] = col;
        F.depth[pix] = dep;
        if (t.store_stencil) F.stencil[pix] = (uint8_t)st;
    }
    uint32_t *const hc = F.host_color;
    float *const hd = F.host_depth;
    uint8_t *const hs = F.host_stencil;
    if (!rows) {
        if (!t.in_fb()) return;
        if (hc) hc[pix] = col;
        if (hd) hd[pix] = dep;
        if (hs) hs[pix] = (uint8_t)st;
        return;
    }
    if (!hc && !hd && !hs) return;
    const int i = (t.py() & (TS - 1)) * TS + (t.px() & (TS - 1));
    if (hc) rows->col[i] = col;
    if (hd) rows->dep[i] = dep;
    if (hs) rows->st[i] = (uint8_t)st;
    __syncthreads();
    const int j = (int)threadIdx.x, px = (t.wx0 & ~(TS - 1)) + j % TS, py = (t.wy0 & ~(TS - 1)) + j / TS;
    if (px >= W || py >= H) return;
    const size_t to = (size_t)py * W + px;
    if (hc) hc[to] = rows->col[j];
    if (hd) hd[to] = rows->dep[j];
    if (hs) hs[to] = rows->st[j];
}

// The pass made more records or pairs than it has room for: every framebuffer is left alone. (One
// load: the two totals are neighbours.)
__device__ __forceinline__ bool over_capacity(const TileArgs &A)
{
    if (!A.guard) return false;
    const uint2 n = __ldg(reinterpret_cast<const uint2 *>(A.guard));
    return n.x > A.records_cap || n.y > A.pairs_cap;
}

// A tile without records or clears has nothing to do, unless its frame is read back.
__device__ __forceinline__ bool idle_tile(const DevFrame &F, uint32_t count)
{
    return count == 0 && F.nclears == 0 && !F.cleared && !F.host_color && !F.host_depth && !F.host_stencil;
}

// ------------------------------------------------------------------ coverage of a block

// Words of a staged record, wherever the stage keeps them.
struct EdgeWords {
    float4 q0, q1, q2, q12, q13;  // x0 y0 x1 y1 | x2 y2 box min | box max area 1/area | flags and edge differences
};

// A triangle against the pixels [xl, xh] x [yl, yh] of a block: can any be covered, must all
// be. The per-pixel test of edge k (raster.c:534-540) is p >= r with p = (x - ax) * A and r =
// (y - ay) * B as floats (a difference of floats has the sign of their order), both sides
// negated for a negative area; p is monotone in x and r in y, rounding included, so their
// extremes over the rectangle are at its corners, exactly.
__device__ __forceinline__ void corner_test(const EdgeWords &w, int xl, int xh, int yl, int yh, bool &any, bool &all)
{
    const float sg = w.q2.z > 0.0f ? 1.0f : -1.0f;
    any = w.q2.z > 0.0f || w.q2.z < 0.0f;
    all = any;
    const float fxl = (float)xl, fxh = (float)xh, fyl = (float)yl, fyh = (float)yh;
    const float ax[3] = {w.q0.z, w.q1.x, w.q0.x}, ay[3] = {w.q0.w, w.q1.y, w.q0.y};
    const float ea[3] = {w.q12.y, w.q12.w, w.q13.y}, eb[3] = {w.q12.z, w.q13.x, w.q13.z};
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const float a = ea[k] * sg, b = eb[k] * sg;
        const float p0 = (fxl - ax[k]) * a, p1 = (fxh - ax[k]) * a;
        const float r0 = (fyl - ay[k]) * b, r1 = (fyh - ay[k]) * b;
        any = any && fmaxf(p0, p1) >= fminf(r0, r1);
        all = all && fminf(p0, p1) >= fmaxf(r0, r1);
    }
}

// the coverage test of a triangle at one pixel of its box
__device__ __forceinline__ bool tri_covers(const EdgeWords &w, float fpx, float fpy)
{
    const float e0 = (fpx - w.q0.z) * w.q12.y - (fpy - w.q0.w) * w.q12.z;
    const float e1 = (fpx - w.q1.x) * w.q12.w - (fpy - w.q1.y) * w.q13.x;
    const float e2 = (fpx - w.q0.x) * w.q13.y - (fpy - w.q0.y) * w.q13.z;
    return (w.q2.z > 0 && e0 >= 0 && e1 >= 0 && e2 >= 0) || (w.q2.z < 0 && e0 <= 0 && e1 <= 0 && e2 <= 0);
}

// the record's box at one pixel
__device__ __forceinline__ bool box_holds(const EdgeWords &w, int px, int py)
{
    return px >= __float_as_int(w.q1.z) && px <= __float_as_int(w.q2.x) && py >= __float_as_int(w.q1.w) &&
           py <= __float_as_int(w.q2.y);
}

// the box's pixels in the block at (wx0, wy0), bit 8 * row + column
__device__ __forceinline__ uint32_t box_mask(const EdgeWords &w, int wx0, int wy0)
{
    const int c0 = max(__float_as_int(w.q1.z) - wx0, 0), c1 = min(__float_as_int(w.q2.x) - wx0, 7);
    const int r0 = max(__float_as_int(w.q1.w) - wy0, 0), r1 = min(__float_as_int(w.q2.y) - wy0, 3);
    if (c0 > c1 || r0 > r1) return 0u;
    const uint32_t cols = (0xFFu >> (7 - c1)) & (0xFFu << c0);
    return (cols * 0x01010101u) & (0xFFFFFFFFu >> (8 * (3 - r1))) & (0xFFFFFFFFu << (8 * r0));
}

// A triangle's covered pixels of the block (the box aside): the per-pixel test in the form of
// corner_test, 32 pixels from 24 + 12 products.
__device__ __forceinline__ uint32_t tri_mask(const EdgeWords &w, int wx0, int wy0)
{
    const float sg = w.q2.z > 0.0f ? 1.0f : -1.0f;
    const float ax[3] = {w.q0.z, w.q1.x, w.q0.x}, ay[3] = {w.q0.w, w.q1.y, w.q0.y};
    const float ea[3] = {w.q12.y, w.q12.w, w.q13.y}, eb[3] = {w.q12.z, w.q13.x, w.q13.z};
    float p[3][8];
#pragma unroll
    for (int k = 0; k < 3; k++)
#pragma unroll
        for (int c = 0; c < 8; c++) p[k][c] = ((float)(wx0 + c) - ax[k]) * (ea[k] * sg);
    uint32_t m = 0;
#pragma unroll
    for (int r = 0; r < 4; r++) {
        float y[3];
#pragma unroll
        for (int k = 0; k < 3; k++) y[k] = ((float)(wy0 + r) - ay[k]) * (eb[k] * sg);
#pragma unroll
        for (int c = 0; c < 8; c++)
            if (p[0][c] >= y[0] && p[1][c] >= y[1] && p[2][c] >= y[2]) m |= 1u << (8 * r + c);
    }
    return m;
}

// ------------------------------------------------------------------ colour

// The colour stages of a fragment (raster.c:582-705): colour interpolation (or the flat
// colour), per-fragment lighting, texturing with the alpha test and texture environment,
// fog. r4: the record's 16-byte words, staged or in memory. Returns false when the alpha test
// discards the fragment.
template <bool TEX, bool EYE>
__device__ __forceinline__ bool frag_color(const DevRaster &R, uint32_t ctl, const float4 *r4, const float *e,
                                           bool have_eye, float b0, float b1, float b2, float4 &c)
{
    const FragState &S = R.fs;
    const float4 c2 = r4[7];  // C2
    if (ctl & FC_FLAT) {
        c = c2;
    } else {
        const float4 c0 = r4[5], c1 = r4[6];  // C0, C1
        c = add4(add4(scale4(c0, b0), scale4(c1, b1)), scale4(c2, b2));
    }
    if (EYE && have_eye) {
        const mtgl_raster_state &rs = R.rs;
        if (rs.lighting) {
            const bool back = (__float_as_uint(r4[12].x) & 1u) != 0;
            const bool phong = rs.shade_model == GL_PHONG;
            if (phong || (back && rs.lit.two_side)) {
                float3 ep = make_float3(e[0] * b0 + e[6] * b1 + e[12] * b2, e[1] * b0 + e[7] * b1 + e[13] * b2,
                                        e[2] * b0 + e[8] * b1 + e[14] * b2);
                float3 en = make_float3(e[3] * b0 + e[9] * b1 + e[15] * b2, e[4] * b0 + e[10] * b1 + e[16] * b2,
                                        e[5] * b0 + e[11] * b1 + e[17] * b2);
                const mtgl_material *mat = &rs.lit.front;
                if (back && rs.lit.two_side) {
                    en = make_float3(en.x * -1.0f, en.y * -1.0f, en.z * -1.0f);
                    mat = &rs.lit.back;
                }
                c = compute_lighting(rs.lit, ep, en, *mat);
            }
        }
    }
    if (TEX && (ctl & FC_TEXTURE)) {
        float u, v;
        const float4 q4 = r4[4];  // W0 W1 W2 LOD
        if (!(ctl & FC_AFFINE_UV)) {
            const float4 q9 = r4[9], q10 = r4[10];  // UV2 UW0 VW0 | UW1 VW1 UW2 VW2
            const float uow = b0 * q9.z + b1 * q10.x + b2 * q10.z;
            const float vow = b0 * q9.w + b1 * q10.y + b2 * q10.w;
            const float oow = b0 * q4.x + b1 * q4.y + b2 * q4.z;
            const float w = 1.0f / oow;
            u = uow * w;
            v = vow * w;
        } else {
            const float4 q8 = r4[8], q9 = r4[9];  // UV0 UV1 | UV2 ..
            u = b0 * q8.x + b1 * q8.z + b2 * q9.x;
            v = b0 * q8.y + b1 * q8.w + b2 * q9.y;
        }
        const float4 tc = sample_lod(S, u, v, q4.w);
        // the alpha test applies to textured fragments only (raster.c:639-643)
        if ((ctl & FC_ALPHA) && !cmp_pass(__ldg(&S.alpha_func), tc.w, __ldg(&S.alpha_ref))) return false;
        switch (__ldg(&S.tex_env_mode)) {
        case GL_REPLACE: c = tc; break;
        case GL_DECAL: c = lerp_rgb(c, tc, tc.w); break;
        case GL_BLEND: {
            const float4 ec = __ldg(reinterpret_cast<const float4 *>(S.tex_env_color));
            c = make_float4(c.x * (1.0f - tc.x) + ec.x * tc.x, c.y * (1.0f - tc.y) + ec.y * tc.y,
                            c.z * (1.0f - tc.z) + ec.z * tc.z, c.w * tc.w);
            break;
        }
        case GL_ADD: c = make_float4(c.x + tc.x, c.y + tc.y, c.z + tc.z, c.w * tc.w); break;
        default: c = mul4(c, tc); break;
        }
    }
    if (ctl & FC_FOG) {
        const float4 q11 = r4[11];                                   // EZ0 EZ1 EZ2
        const float4 g3 = __ldg(reinterpret_cast<const float4 *>(&S) + 3);  // .z mode, .w density
        const float4 g4 = __ldg(reinterpret_cast<const float4 *>(&S) + 4);  // .x start, .y end
        const float4 fcol = __ldg(reinterpret_cast<const float4 *>(S.fog_color));
        const float fc = b0 * q11.x + b1 * q11.y + b2 * q11.z;
        c = lerp_rgb(fcol, c, fog_factor(__float_as_uint(g3.z), g3.w, g4.x, g4.y, fc));
    }
    return true;
}

// The barycentrics of the pixel in a triangle record, as the coverage test computes them.
__device__ __forceinline__ void tri_bary(const float4 *r4, float fpx, float fpy, float &b0, float &b1, float &b2)
{
    const float4 q0 = __ldg(r4 + 0), q1 = __ldg(r4 + 1), q2 = __ldg(r4 + 2), q12 = __ldg(r4 + 12),
                 q13 = __ldg(r4 + 13);
    const float e0 = (fpx - q0.z) * q12.y - (fpy - q0.w) * q12.z;
    const float e1 = (fpx - q1.x) * q12.w - (fpy - q1.y) * q13.x;
    const float e2 = (fpx - q0.x) * q13.y - (fpy - q0.y) * q13.z;
    b0 = e0 * q2.w;
    b1 = e1 * q2.w;
    b2 = e2 * q2.w;
}

// The colour a deferred fragment writes (below): its colour stages, clamped and packed (its
// raster state has no blend and writes every channel).
template <bool TEX, bool EYE>
__device__ __forceinline__ uint32_t pending_color(const TileArgs &A, uint32_t ridx, bool have_eye, float fpx,
                                                  float fpy)
{
    const float4 *r4 = reinterpret_cast<const float4 *>(A.records + (size_t)ridx * kRecWords);
    const float *e = have_eye ? A.eye_records + (size_t)ridx * kEyeWords : nullptr;
    float b0, b1, b2;
    tri_bary(r4, fpx, fpy, b0, b1, b2);
    const float4 q11 = __ldg(r4 + 11);
    const DevRaster &R = A.rasters[min(__float_as_uint(q11.w), A.nrasters - 1)];
    float4 c;
    frag_color<TEX, EYE>(R, __ldg(&R.fs.ctl), r4, e, have_eye, b0, b1, b2, c);
    return pack_rgba(c.x, c.y, c.z, c.w);
}

// ------------------------------------------------------------------ points and lines

// The pixel state a point or line fragment updates (no stencil: the reference's point and
// line paths never touch it).
struct PixelOut {
    uint32_t col;
    float dep;
    uint32_t flags;  // bit 0: a fragment; bit 1: depth written
};

// write_line_pixel (raster.c:86-104) and the pixel loop of draw_points (raster.c:1140-1160) past
// the depth test: blend with the stored colour, depth write, masked colour write. ctl: the
// record's enables.
__device__ __forceinline__ PixelOut point_ops(const FragState &S, uint32_t ctl, float depth, float4 c, uint32_t col,
                                              float dep)
{
    PixelOut o{col, dep, 1u};
    if (ctl & FC_BLEND) c = blend(__ldg(&S.blend_src), __ldg(&S.blend_dst), c, unpack_rgba(col));
    if (ctl & FC_DEPTH_WRITE) {
        o.dep = depth;
        o.flags |= 2u;
    }
    if (ctl & FC_MASK_ALL) o.col = pack_rgba(c.x, c.y, c.z, c.w);
    else if (!(ctl & FC_MASK_NONE)) o.col = masked_write(__ldg(&S.color_mask), col, c);
    return o;
}

// A line record's pixels of the block (the box aside, which holds the framebuffer and scissor
// limits). The Bresenham step reaching a pixel in closed form: for an x-major line (|dx| > |dy|)
// step k sits at x0 + sx*k, y0 + sy*floor((2|dy|k + |dx| - 1) / (2|dx|)); for a y-major one the
// roles swap; each step writes a run of `lw` pixels across the major axis. That reproduces
// draw_line_full's loop exactly (tests/test_arith.py checks it against the loop over every
// |dx|, |dy| <= 130). One division per column (row) of the block; I: int32 where every value
// fits, which a line inside a framebuffer does.
template <class I, class U>
__device__ __forceinline__ uint32_t line_mask_of(I x0, I y0, I x1, I y1, I lw, int wx0, int wy0)
{
    const I half = lw / 2, dx = x1 - x0, dy = y1 - y0;
    const I adx = dx < 0 ? -dx : dx, ady = dy < 0 ? -dy : dy;
    const I sx = dx < 0 ? -1 : 1, sy = dy < 0 ? -1 : 1;
    uint32_t m = 0;
    if (adx > ady) {
        for (int c = 0; c < 8; c++) {
            const I k = ((I)(wx0 + c) - x0) * sx;
            if (k < 0 || k > adx) continue;
            const I y = y0 + sy * (I)((U)(2 * ady * k + adx - 1) / (U)(2 * adx));
            const I r0 = y - half - wy0, r1 = y + lw - half - 1 - wy0;
            if (r1 < 0 || r0 > 3) continue;
            const uint32_t rows = (0xFu >> (3 - (int)(r1 < 3 ? r1 : 3))) & (0xFu << (int)(r0 > 0 ? r0 : 0));
            m |= ((rows * 0x00204081u) & 0x01010101u) << c;  // bit r of rows to bit 8 * r
        }
    } else {
        for (int r = 0; r < 4; r++) {
            I x = x0;
            if (ady > 0) {
                const I k = ((I)(wy0 + r) - y0) * sy;
                if (k < 0 || k > ady) continue;
                x = x0 + sx * (I)((U)(2 * adx * k + ady - 1) / (U)(2 * ady));
            } else if ((I)(wy0 + r) != y0) {
                continue;
            }
            const I c0 = x - half - wx0, c1 = x + lw - half - 1 - wx0;
            if (c1 < 0 || c0 > 7) continue;
            m |= ((0xFFu >> (7 - (int)(c1 < 7 ? c1 : 7))) & (0xFFu << (int)(c0 > 0 ? c0 : 0))) << (8 * r);
        }
    }
    return m;
}
static __device__ __noinline__ uint32_t line_mask(const float4 &q0, int lw, int wx0, int wy0)
{
    const int x0 = __float_as_int(q0.x), y0 = __float_as_int(q0.y), x1 = __float_as_int(q0.z), y1 = __float_as_int(q0.w);
    // |coordinates| < 2^14 leaves 2 |dy| k + |dx| below 2^32 (and 2^31: |dx|, |dy| < 2^15)
    auto small = [](int v) { return v > -(1 << 14) && v < (1 << 14); };
    if (small(x0) && small(y0) && small(x1) && small(y1) && small(lw))
        return line_mask_of<int32_t, uint32_t>(x0, y0, x1, y1, lw, wx0, wy0);
    return line_mask_of<int64_t, uint64_t>(x0, y0, x1, y1, lw, wx0, wy0);
}

// Steps to a line's pixel and in all: along x for an x-major line, else along y.
template <class I>
__device__ __forceinline__ void line_step(I x0, I y0, I x1, I y1, int px, int py, int32_t &k, int32_t &total)
{
    const I dx = x1 - x0, dy = y1 - y0;
    const I adx = dx < 0 ? -dx : dx, ady = dy < 0 ? -dy : dy;
    k = (int32_t)(adx > ady ? (dx < 0 ? x0 - px : px - x0) : (ady > 0 ? (dy < 0 ? y0 - py : py - y0) : 0));
    total = (int32_t)(adx > ady ? adx : ady);
}

// One pixel a point or line record covers: with the step's t, its colour, depth, texel and fog.
// Where many short lines meet (a mesh's pole) a pixel takes hundreds of them one after another, and
// the latency of this function bounds the launch: the enables and the depth function come with the
// record, the depth test is first (nothing before it has an effect), and the steps are 32-bit (a
// wireframe sphere with its points, whole passes: 417 -> 388 us).
static __device__ __noinline__ PixelOut shade_prim(const TileArgs &A, const float4 *q, int px, int py, uint32_t col,
                                                   float dep)
{
    const PixelOut none{col, dep, 0u};
    const float4 q0 = q[0], q3 = q[3];
    const uint32_t flags = __float_as_uint(q[12].x), ctl = flags >> kRecCtlShift;
    const uint32_t func = GL_NEVER + ((flags >> kRecDepthFuncShift) & 7u);
    const DevRaster &R = A.rasters[min(__float_as_uint(q[11].w), A.nrasters - 1)];
    const FragState &S = R.fs;
    if (((flags >> kRecTypeShift) & 3u) == REC_POINT) {
        if ((ctl & FC_DEPTH) && !cmp_pass(func, q3.x, dep)) return none;
        return point_ops(S, ctl, q3.x, q[5], col, dep);
    }
    const int x0 = __float_as_int(q0.x), y0 = __float_as_int(q0.y), x1 = __float_as_int(q0.z), y1 = __float_as_int(q0.w);
    auto small = [](int v) { return v > -(1 << 29) && v < (1 << 29); };
    int32_t k, total;
    if (small(x0) && small(y0) && small(x1) && small(y1)) line_step<int32_t>(x0, y0, x1, y1, px, py, k, total);
    else line_step<int64_t>(x0, y0, x1, y1, px, py, k, total);
    const float t = (float)k / (float)(total == 0 ? 1 : total);
    const float z = q3.x + t * (q3.y - q3.x);
    const float u01 = (z + 1.0f) * 0.5f;
    const float depth = (ctl & FC_DEFAULT_RANGE) ? u01 : map_depth_range(u01, R.rs.depth_near, R.rs.depth_far);
    if ((ctl & FC_DEPTH) && !cmp_pass(func, depth, dep)) return none;
    float4 c = lerp_col(q[5], q[6], t);
    // the reference never leaves its loop when the alpha test fails (raster.c:175, 183 skip the
    // Bresenham step); here the pixel is dropped
    if (ctl & FC_TEXTURE) {
        const float4 q8 = q[8];
        const float u = q8.x + t * (q8.z - q8.x);
        const float v = q8.y + t * (q8.w - q8.y);
        const float4 tc = sample_lod(S, u, v, 0.0f);
        if ((ctl & FC_ALPHA) && !cmp_pass(__ldg(&S.alpha_func), tc.w, __ldg(&S.alpha_ref))) return none;
        c = make_float4(c.x * tc.x, c.y * tc.y, c.z * tc.z, c.w * tc.w);
    } else if ((ctl & FC_ALPHA) && !cmp_pass(__ldg(&S.alpha_func), c.w, __ldg(&S.alpha_ref))) {
        return none;
    }
    if (ctl & FC_FOG) {
        const float4 q11 = q[11];
        c = lerp_rgb(__ldg(reinterpret_cast<const float4 *>(S.fog_color)), c,
                     fog_factor(S.fog_mode, S.fog_density, S.fog_start, S.fog_end, -(q11.x + t * (q11.y - q11.x))));
    }
    return point_ops(S, ctl, depth, c, col, dep);
}

// ------------------------------------------------------------------ triangles

// One covered fragment of rasterize_triangle_smooth's pixel loop (raster.c:534-722) for this
// thread's pixel. Returns true when it wrote the depth buffer. TEX / EYE compile the
// texturing and per-fragment lighting stages in only for passes that use them.
//
// DEFER (deferred colour): in a pass whose every record is a filled triangle whose raster
// state has no blend, writes all four colour channels or none, and cannot have a fragment
// discarded by the alpha test (untextured, or the test off), no fragment reads the stored
// colour, and each fragment that writes colour replaces it. So only the tests, stencil and
// depth writes run per fragment; the pixel keeps the record of the last fragment that
// wrote colour, and its colour stages run once, when the tile is written back. The stored
// colour comes out exactly as if every fragment had been shaded in turn.
template <bool TEX, bool EYE, bool DEFER>
__device__ __forceinline__ bool shade_tri(const TileArgs &A, const float4 *q, uint32_t ridx, bool have_eye, float fpx,
                                          float fpy, uint32_t &col, float &dep, uint32_t &st, uint32_t &pend)
{
    const float4 q0 = q[0], q1 = q[1], q2 = q[2], q3 = q[3], q12 = q[12], q13 = q[13];
    // edge_function at the integer pixel position (raster.c:299-302, 534-536)
    const float e0 = (fpx - q0.z) * q12.y - (fpy - q0.w) * q12.z;
    const float e1 = (fpx - q1.x) * q12.w - (fpy - q1.y) * q13.x;
    const float e2 = (fpx - q0.x) * q13.y - (fpy - q0.y) * q13.z;
    const float inv_area = q2.w;
    const float b0 = e0 * inv_area, b1 = e1 * inv_area, b2 = e2 * inv_area;
    // the raster state, only where a stage reads more than the record carries
    auto raster = [&]() -> const DevRaster & { return A.rasters[min(__float_as_uint(q[11].w), A.nrasters - 1)]; };
    // the enables and the depth function come with the record's flags; the other operands are
    // loaded as the stages need them (from one cached line, to keep few registers live)
    const uint32_t rflags = __float_as_uint(q12.x);
    const uint32_t ctl = (rflags >> kRecCtlShift) & 0xFFFu;
    const float z = b0 * q3.x + b1 * q3.y + b2 * q3.z;
    const float t = (z + 1.0f) * 0.5f;
    const float depth =
        (ctl & FC_DEFAULT_RANGE) ? t : map_depth_range(t, raster().rs.depth_near, raster().rs.depth_far);

    uint32_t sv = 0;
    if (ctl & FC_STENCIL) {
        const FragState &S = raster().fs;
        const uint4 g = __ldg(reinterpret_cast<const uint4 *>(&S) + 1);  // func, ref, mask, writemask
        sv = st;
        if (!stencil_pass(g.x, (int32_t)g.y, g.z, sv)) {
            st = stencil_write(st, stencil_apply(__ldg(&S.stencil_fail), sv, (int32_t)g.y), g.w);
            return false;
        }
    }
    if ((ctl & FC_DEPTH) && !cmp_pass(GL_NEVER + ((rflags >> kRecDepthFuncShift) & 7u), depth, dep)) {
        if (ctl & FC_STENCIL) {
            const FragState &S = raster().fs;
            st = stencil_write(st, stencil_apply(__ldg(&S.stencil_zfail), sv, __ldg(&S.stencil_ref)),
                               __ldg(&S.stencil_writemask));
        }
        return false;
    }
    if (ctl & FC_STENCIL) {
        const FragState &S = raster().fs;
        st = stencil_write(st, stencil_apply(__ldg(&S.stencil_zpass), sv, __ldg(&S.stencil_ref)),
                           __ldg(&S.stencil_writemask));
    }

    if (DEFER) {
        if (ctl & FC_MASK_ALL) pend = ridx;  // this fragment's colour replaces the pixel's
        if (ctl & FC_DEPTH_WRITE) {
            dep = depth;
            return true;
        }
        return false;
    }
    const DevRaster &R = raster();
    const FragState &S = R.fs;
    float4 c;
    const float *e = have_eye ? A.eye_records + (size_t)ridx * kEyeWords : nullptr;
    if (!frag_color<TEX, EYE>(R, ctl, q, e, have_eye, b0, b1, b2, c)) return false;
    bool wrote = false;
    if (ctl & FC_DEPTH_WRITE) {
        dep = depth;
        wrote = true;
    }
    if (ctl & FC_BLEND) c = blend(__ldg(&S.blend_src), __ldg(&S.blend_dst), c, unpack_rgba(col));
    if (ctl & FC_MASK_ALL) col = pack_rgba(c.x, c.y, c.z, c.w);
    else if (!(ctl & FC_MASK_NONE)) col = masked_write(__ldg(&S.color_mask), col, c);
    return wrote;
}

// ------------------------------------------------------------------ the ordered kernel

// Records staged at a time. A block takes part of them, and its rounds are as many as its deepest
// pixel's records: of 64 records the deepest pixel is nearer the mean than of 32, and one set of
// masks serves both halves (a million blended triangles at 1080p: 947 -> 791 us). Textured passes
// read texels through the L1 that 64 records would take (600 sprites in 4K, whole passes: 982 us with 32,
// 1019 with 64); the other tile sizes have no shared memory for 64.
template <int TS, bool TEX>
__host__ __device__ constexpr int step_records()
{
    return TS == 16 && !TEX ? 64 : 32;
}
constexpr int kPickIndex = 0xFF, kPickAll = 0x100;  // a listed record: its place in the chunk, covers the block
constexpr int kStepWords = 17;    // 16-byte words per staged record: 15 and its index, stride free of bank conflicts
constexpr int kFewRecords = 6;    // up to this many left in a block: test each at every pixel; more go by masks

// 64 registers and 1024 resident threads per SM (the fragment pipeline spills at 48).
template <int TS>
constexpr int tile_min_blocks()
{
    return TS == 32 ? 1 : 1024 / (TS * TS);
}

// Depths as ordered integers, the zeros equal: a record is hidden when its key is at least the
// largest stored depth's (one less under GL_LEQUAL). Above INT32_MIN, the key of what is never hidden.
__device__ __forceinline__ int far_key(float depth) { return ordered_key(depth + 0.0f); }
__device__ __forceinline__ int block_far_key(float dep, bool in_fb)
{
    return __reduce_max_sync(0xffffffffu, in_fb ? far_key(dep) : INT32_MIN);
}

template <int TS, bool TEX, bool EYE, bool DEFER>
__global__ void __launch_bounds__(TS *TS, tile_min_blocks<TS>()) k_tile(TileArgs A)
{
    constexpr int kThreads = TS * TS, kStep = step_records<TS, TEX>();  // a pick's index fits kPickIndex
    __shared__ float4 s_rec[2][kStep * kStepWords];
    // a warp's records of a chunk: index and kPickAll, hiding far key; a chunk of 32 needs no list,
    // its records stay with their lanes
    constexpr bool kListed = kStep > 32;
    __shared__ int2 s_pick[kListed ? kThreads / 32 : 1][kStep];
    int2 *const pick = s_pick[kListed ? threadIdx.x >> 5 : 0];

    const bool over = over_capacity(A);  // waited for with the first tile's words
    const int lane = threadIdx.x & 31;
    const bool have_eye = EYE && A.eye_records != nullptr;
    uint32_t frags = 0;
    for (uint32_t it = blockIdx.x; it < A.ntiles; it += gridDim.x) {
        const uint32_t tile = A.order ? A.order[it] : it;
        const uint32_t count = A.tile_count[tile], start = A.tile_start[tile];
        const DevFrame &F = A.frames[A.tile_frame ? A.tile_frame[tile] : 0u];
        if (over) return;
        if (idle_tile(F, count)) continue;
        if (!debug_check(A.debug, (uint64_t)start + count <= A.entries_cap, DBG_TILE_ENTRY)) continue;
        if (it != blockIdx.x) __syncthreads();  // the previous tile's records are done with

        // stage records [base, base + kStep) of the list: 16 threads per record, one word each
        auto stage = [&](uint32_t base, int buf) {
            const uint32_t m = min((uint32_t)kStep, count - base);
            for (uint32_t i = threadIdx.x; i < 16 * m; i += kThreads) {
                const uint32_t e = i >> 4, w = i & 15u;
                uint32_t idx = __ldg(A.tile_vals + start + base + e);
                if (!debug_check(A.debug, idx < A.records_cap, DBG_TILE_RECORD)) idx = 0;
                float4 *d = s_rec[buf] + e * kStepWords;
                if (w == 15u) d[15].x = __uint_as_float(idx);
                else if (TEX || !(w == 4u || (w >= 8u && w <= 10u)))  // texturing's words
                    cp_async16(d + w, reinterpret_cast<const float4 *>(A.records + (size_t)idx * kRecWords) + w);
            }
        };
        if (count) stage(0, 0);
        cp_async_commit();

        const TilePixel t = open_tile<TS>(A, F, tile, A.any_stencil != 0);
        uint32_t col = t.col, st = t.st, pend = kNoPending;
        float dep = t.dep;
        const float fpx = (float)t.px(), fpy = (float)t.py();
        // hierarchical z: the block's largest stored depth
        int far = block_far_key(dep, t.in_fb());
        int buf = 0;
        for (uint32_t base = 0; base < count; base += kStep, buf ^= 1) {
            cp_async_wait_all();
            __syncthreads();
            if (base + kStep < count) {
                stage(base + kStep, buf ^ 1);
                cp_async_commit();
            }
            if (t.wx1 < t.wx0 || t.wy1 < t.wy0) continue;  // the block lies outside the framebuffer
            const int m = (int)min((uint32_t)kStep, count - base);
            const float4 *rec = s_rec[buf];
            // Lane j takes record base + s0 + j: can it cover a pixel of the block, does it cover all,
            // and can a fragment pass the depth test (rejected by the bound over the block against the
            // largest stored depth, unless a record of the chunk before it may raise depths). Those
            // left are listed in order, with the far key from which on they are hidden.
            int n = 0;
            bool raised = false;
            uint32_t listed = 0;
            int2 mine;
#pragma unroll 1
            for (int s0 = 0; s0 < m; s0 += 32) {
                bool take = false, all = false;
                uint32_t flags = 0;
                int hide = INT32_MIN;  // never
                if (s0 + lane < m) {
                    const float4 *q = rec + (s0 + lane) * kStepWords;
                    const EdgeWords w{q[0], q[1], q[2], q[12], q[13]};
                    flags = __float_as_uint(w.q12.x);
                    const int mnx = __float_as_int(w.q1.z), mny = __float_as_int(w.q1.w);
                    const int xl = max(t.wx0, mnx), xh = min(t.wx1, __float_as_int(w.q2.x));
                    const int yl = max(t.wy0, mny), yh = min(t.wy1, __float_as_int(w.q2.y));
                    take = xl <= xh && yl <= yh;
                    if (take && ((flags >> kRecTypeShift) & 3u) == REC_TRI) {
                        corner_test(w, xl, xh, yl, yh, take, all);
                        all = all && xl == t.wx0 && xh == t.wx1 && yl == t.wy0 && yh == t.wy1;
                        const uint32_t zc = (flags >> 1) & 3u;
                        if (zc == ZC_LESS || zc == ZC_LEQUAL) {
                            const float lo = fmaxf(q[3].w, depth_plane_bound(q[14], mnx, mny, xl, xh, yl, yh));
                            if (lo == lo) hide = far_key(lo) - (zc == ZC_LESS ? 0 : 1);
                        } else if (zc == ZC_NEVER) {
                            hide = INT32_MAX;
                        }
                    }
                }
                const uint32_t raise = __ballot_sync(0xffffffffu, (flags & kFlagRaisesDepth) != 0);
                if (!raised && (raise & ((1u << lane) - 1u)) == 0 && hide >= far) take = false;
                raised = raised || raise != 0;
                listed = __ballot_sync(0xffffffffu, take);
                mine = make_int2((s0 + lane) | (take && all ? kPickAll : 0), hide);
                if (kListed && take) pick[n + __popc(listed & ((1u << lane) - 1u))] = mine;
                n += __popc(listed);
            }
            __syncwarp();
            auto record = [&](int b0, int j) { return rec + (kListed ? pick[b0 + j].x & kPickIndex : j) * kStepWords; };
            for (int b0 = 0; b0 < n; b0 += 32) {
                if (kListed) {
                    listed = __ballot_sync(0xffffffffu, b0 + lane < n);
                    mine = b0 + lane < n ? pick[b0 + lane] : make_int2(0, INT32_MIN);
                }
                // the listed records of this lane's pixel, in order
                uint32_t cov = __ballot_sync(0xffffffffu, (mine.x & kPickAll) != 0);
                uint32_t todo = listed & ~cov;
                if (!t.in_fb()) cov = 0;
                if (__popc(todo) <= kFewRecords) {
                    for (; todo; todo &= todo - 1) {
                        const int j = __ffs(todo) - 1;
                        const float4 *q = record(b0, j);
                        const EdgeWords v{q[0], q[1], q[2], q[12], q[13]};
                        bool in = box_holds(v, t.px(), t.py());
                        const uint32_t type = (__float_as_uint(v.q12.x) >> kRecTypeShift) & 3u;
                        if (type == REC_TRI) in = in && tri_covers(v, fpx, fpy);
                        else if (!DEFER && type == REC_LINE)
                            in = in && ((line_mask(v.q0, __float_as_int(v.q1.x), t.wx0, t.wy0) >> lane) & 1u);
                        if (in) cov |= 1u << j;
                    }
                } else {
                    uint32_t mask = 0;
                    if ((todo >> lane) & 1u) {
                        const float4 *q = rec + (mine.x & kPickIndex) * kStepWords;
                        const EdgeWords w{q[0], q[1], q[2], q[12], q[13]};
                        mask = box_mask(w, t.wx0, t.wy0);
                        const uint32_t type = (__float_as_uint(w.q12.x) >> kRecTypeShift) & 3u;
                        if (type == REC_TRI) mask &= tri_mask(w, t.wx0, t.wy0);
                        else if (!DEFER && type == REC_LINE) mask &= line_mask(w.q0, __float_as_int(w.q1.x), t.wx0, t.wy0);
                    }
                    cov |= warp_transpose(mask);
                }
                frags += __popc(cov);
                while (__any_sync(0xffffffffu, cov != 0)) {
                    bool wrote = false;
                    if (cov) {
                        const float4 *q = record(b0, __ffs(cov) - 1);
                        cov &= cov - 1;
                        if (DEFER || ((__float_as_uint(q[12].x) >> kRecTypeShift) & 3u) == REC_TRI) {
                            wrote = shade_tri<TEX, EYE, DEFER>(A, q, __float_as_uint(q[15].x), have_eye, fpx, fpy, col,
                                                               dep, st, pend);
                        } else {
                            const PixelOut po = shade_prim(A, q, t.px(), t.py(), col, dep);
                            col = po.col;
                            dep = po.dep;
                            wrote = (po.flags & 2u) != 0;
                        }
                    }
                    if (__any_sync(0xffffffffu, wrote)) {
                        far = block_far_key(dep, t.in_fb());
                        // while depths only fall, drop what they now hide
                        if (!raised) cov &= ~__ballot_sync(0xffffffffu, mine.y >= far);
                    }
                }
            }
        }
        if (DEFER && pend != kNoPending) col = pending_color<TEX, EYE>(A, pend, have_eye, fpx, fpy);
        close_tile<TS>(A, F, t, col, dep, st, nullptr);
    }
    if (A.fragments) {
        const uint32_t fw = __reduce_add_sync(0xffffffffu, frags);
        if (lane == 0 && fw) atomicAdd(A.fragments, (unsigned long long)fw);
    }
}

// One CTA per tile, or A.ctas of them that step through the tiles.
template <class K>
inline void launch_tiles(K kernel, const TileArgs &a, int threads, cudaStream_t s)
{
    kernel<<<a.ctas ? (unsigned)std::min<uint32_t>((uint32_t)a.ctas, a.ntiles) : a.ntiles, threads, 0, s>>>(a);
}

template <class K>
inline int tiles_per_sm(K kernel, int threads)
{
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, 0) != cudaSuccess) n = 1;
    return n > 0 ? n : 1;
}

// Runs `f` with the kernel of the pass's tile size and stages: f(kernel, threads).
template <bool DEFER, class F>
auto with_tile_kernel(const TileArgs &a, F f)
{
    const bool eye = a.eye_records != nullptr;
    auto pick = [&](auto none, auto tex, auto eyes, auto both_, int threads) {
        return f(a.any_texture ? (eye ? both_ : tex) : (eye ? eyes : none), threads);
    };
    switch (a.tile_shift) {
    case 3: return pick(k_tile<8, false, false, DEFER>, k_tile<8, true, false, DEFER>, k_tile<8, false, true, DEFER>, k_tile<8, true, true, DEFER>, 64);
    case 5: return pick(k_tile<32, false, false, DEFER>, k_tile<32, true, false, DEFER>, k_tile<32, false, true, DEFER>, k_tile<32, true, true, DEFER>, 1024);
    default: return pick(k_tile<16, false, false, DEFER>, k_tile<16, true, false, DEFER>, k_tile<16, false, true, DEFER>, k_tile<16, true, true, DEFER>, 256);
    }
}

// the deferred-colour and the order-free launches (k_tile_defer.cu, k_tile_free.cu), or their
// resident CTAs per SM
int launch_tile_deferred(const TileArgs &a, cudaStream_t s);
int deferred_per_sm(const TileArgs &a);
int launch_tile_free(const TileArgs &a, cudaStream_t s);
int free_per_sm(const TileArgs &a);

}  // namespace mtgl
