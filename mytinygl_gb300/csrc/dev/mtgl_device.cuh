// mtgl_device.cuh — device-side data layout and arithmetic of the GB300 back end.
//
// Every float expression here reproduces the reference's operation order (src/graphics.h,
// src/lighting.h, src/raster.c, src/textures.c) and the translation units are compiled
// with -fmad=false and IEEE division/square root, so each result is the value the
// reference computes on x86-64. Float->int conversions emulate x86-64 cvttss2si (NaN and
// out-of-range give INT32_MIN), which is what the reference's casts compile to.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "GL/gl.h"
#include "mytinygl/mtgl_dev.h"

namespace mtgl {

// ------------------------------------------------------------------ debug bounds checks
//
// A build with MTGL_DEBUG_BOUNDS defined (mytinygl_gb300.build(debug_bounds=True)) checks the
// index of every device-memory access the kernels compute from data (framebuffer pixels,
// triangle records, tile-list entries, tile ids, vertex slots). A failed check never traps:
// it records its site code in the context's status word (the first failure wins; read back
// through mtgl_stats.debug_status) and skips the access. In the ordinary build the checks
// compile to nothing.
enum DebugSite : uint32_t {
    DBG_TILE_PIXEL = 1,    // K4: framebuffer pixel index
    DBG_TILE_RECORD = 2,   // K4: record index from a tile list
    DBG_TILE_ENTRY = 3,    // K4: tile-list position
    DBG_BIN_TILE = 4,      // binning: tile id of a sorted pair
    DBG_VERTEX_SLOT = 5,   // K1: vertex slot
    DBG_SETUP_RECORD = 6,  // K2: record position
    // Not an index check, and recorded by every build: a scan's bounded wait for an earlier
    // tile's sum ran out (never expected; the pass's results are then wrong).
    DBG_SCAN_WAIT = 7,
};
__device__ __forceinline__ bool debug_check(uint32_t *status, bool ok, uint32_t site)
{
#ifdef MTGL_DEBUG_BOUNDS
    if (!ok && status) atomicCAS(status, 0u, site);
    return ok;
#else
    (void)status;
    (void)site;
    (void)ok;
    return true;
#endif
}

// ------------------------------------------------------------------ layout constants

constexpr int kTileShiftMin = 3;     // tile edges of 8, 16 or 32 pixels (one CTA per tile)
constexpr int kTileShiftMax = 5;
constexpr int kTileShiftPlain = 4;   // 16x16 tiles for single-frame passes
constexpr int kRecWords = 60;        // words per triangle record (240 bytes)
constexpr int kEyeWords = 20;        // words per triangle eye-space record (per-fragment lighting)

// Triangle record written by the setup kernel, read by the tile kernel (raster.c:451-529
// inputs plus the per-triangle values rasterize_triangle_smooth derives before its loop).
enum RecField {
    R_X0 = 0, R_Y0, R_X1, R_Y1, R_X2, R_Y2,   // screen vertices as floats of the int coordinates
    R_MINX = 6, R_MINY, R_MAXX, R_MAXY,       // int32 bbox after viewport/scissor/framebuffer clamps
    R_AREA = 10, R_INV_AREA,
    R_Z0 = 12, R_Z1, R_Z2,
    R_DMIN = 15,                              // lower bound of every fragment depth (hierarchical z)
    R_W0 = 16, R_W1, R_W2,                    // 1/w
    R_LOD = 19,
    R_C0 = 20, R_C1 = 24, R_C2 = 28,          // RGBA each
    R_UV0 = 32, R_UV1 = 34, R_UV2 = 36,       // raw texcoords
    R_UW0 = 38, R_VW0, R_UW1, R_VW1, R_UW2, R_VW2,
    R_EZ0 = 44, R_EZ1, R_EZ2,
    R_RASTER = 47,                            // uint32 raster-state index
    R_FLAGS = 48,                             // bit 0 back facing; bits 1-2 depth rejection mode
    R_EA0 = 49, R_EB0, R_EA1, R_EB1, R_EA2, R_EB2,  // per-edge (by-ay), (bx-ax) of edge_function
    R_FRAME = 55,                             // uint32 frame index within the pass's frame table
    // the depth plane over the box, for a per-block depth bound (depth_plane_bound):
    // z at (MINX, MINY), dz/dx, dz/dy, and the margin that makes the bound safe (+inf: none)
    R_ZP0 = 56, R_ZGX, R_ZGY, R_ZM
};

// Depth rejection modes (R_FLAGS bits 1-2). A warp skips a triangle when no fragment of it
// can pass the depth test and a failing fragment has no other effect (stencil test off):
// GL_LESS: min fragment depth >= the warp's max stored depth; GL_LEQUAL: >; GL_NEVER: always.
enum ZCull { ZC_NONE = 0, ZC_LESS = 1, ZC_LEQUAL = 2, ZC_NEVER = 3 };
// R_FLAGS bit 3: the triangle may raise stored depths (depth writes with GL_GREATER,
// GL_GEQUAL, GL_NOTEQUAL or GL_ALWAYS); a warp's max depth taken before it is then no bound.
constexpr uint32_t kFlagRaisesDepth = 8u;

// R_FLAGS bits 4-5: what the record draws. Points and lines reuse the record's words:
//   REC_POINT (draw_points / draw_point_at_screen, raster.c:777-844, 1020-1164): a square
//     R_MINX..R_MAXY (already clamped to the framebuffer and scissor) of one depth R_Z0 and
//     one final colour R_C0 (texture, alpha test and fog applied at setup);
//   REC_LINE (draw_line_full, raster.c:107-241): int endpoints R_X0,R_Y0 / R_X1,R_Y1, width
//     R_X2 (int), NDC z R_Z0/R_Z1, colours R_C0/R_C1, uv R_UV0/R_UV1, eye z R_EZ0/R_EZ1,
//     bbox R_MINX..R_MAXY over the widened line clamped to framebuffer and scissor.
enum RecType { REC_TRI = 0, REC_POINT = 1, REC_LINE = 2 };
constexpr int kRecTypeShift = 4;
// R_FLAGS bits 8-19: the raster state's FragCtl enables; bits 20-22: its depth function -
// GL_NEVER. The tile kernel's tests read them with the edge
// coefficients (same 16-byte word) instead of through the raster state.
constexpr int kRecCtlShift = 8, kRecDepthFuncShift = 20;

// Lower bound of the depth of every fragment a triangle record can write in the rectangle
// [xl, xh] x [yl, yh] of its box (inclusive pixel positions, inside the record's box).
// The record stores a float plane p(x, y) = P0 + GX (x - MINX) + GY (y - MINY) close to the
// exact interpolation Z*(x, y) = sum z_i e_i(x, y) / area, and a margin M covering, for every
// covered pixel of the box, the roundings of the fragment's own z (b_i = e_i * inv_area,
// then the sum), of P0, GX and GY, and of this evaluation (setup_fan_tri derives it). The
// plane's minimum over the rectangle is at the corner the signs of GX and GY pick; the
// depth mapping of the default range, (z + 1) * 0.5, is monotone. With M = +inf (no plane)
// the result is -inf.
__device__ __forceinline__ float depth_plane_bound(const float4 &zp, int minx, int miny, int xl, int xh, int yl,
                                                  int yh)
{
    const float dx = (float)((zp.y >= 0.0f ? xl : xh) - minx);
    const float dy = (float)((zp.z >= 0.0f ? yl : yh) - miny);
    const float z = (zp.x + zp.y * dx) + zp.z * dy - zp.w;
    return (z + 1.0f) * 0.5f;
}

// Upper bound of the same fragment depths, from the same plane: its maximum over the
// rectangle plus the margin, which bounds the errors on either side. +inf without a plane.
__device__ __forceinline__ float depth_plane_upper(const float4 &zp, int minx, int miny, int xl, int xh, int yl,
                                                   int yh)
{
    const float dx = (float)((zp.y >= 0.0f ? xh : xl) - minx);
    const float dy = (float)((zp.z >= 0.0f ? yh : yl) - miny);
    const float z = (zp.x + zp.y * dx) + zp.z * dy + zp.w;
    return (z + 1.0f) * 0.5f;
}

// Float order as unsigned order, reversed: a nearer depth has the larger key, and 0 is beyond
// every depth (the tile occlusion bounds of binning start at zero bytes and take a maximum).
__device__ __forceinline__ uint32_t near_key(float f)
{
    const uint32_t b = __float_as_uint(f);
    return ~(b ^ ((uint32_t)((int32_t)b >> 31) | 0x80000000u));
}

// Post-transform vertices (vertex_t, graphics.h:438-446, without the unused object normal)
// are stored as three streams of 16-byte words, one word per vertex slot each: the clip
// position, the colour, and (u, v, eye z, 0). The count pass of set-up reads only the first.
struct PostVertices {
    float4 *clip;
    float4 *color;
    float4 *uvz;
};
struct __align__(16) PostEye {
    float4 pos_nx;   // eye_pos.xyz, eye_normal.x
    float4 nyz;      // eye_normal.y, eye_normal.z
};

struct DevAttrib {
    const uint8_t *ptr;   // element `base_index` is at ptr
    int64_t base_index;
    uint64_t bytes;       // readable bytes from ptr
    int32_t size, type, stride, enabled;
};

// One draw packet as the kernels see it.
struct DevDraw {
    uint32_t mode;
    int32_t first, count;
    uint32_t index_type;
    const uint8_t *indices;
    int64_t index_min;
    int32_t range_n;       // range mode: vertices index_min .. index_min+range_n-1
    int32_t range_mode;    // 1: slots cover an index range (+1 default slot), 0: one slot per element
    int32_t pos2d;
    DevAttrib pos, color, tex, normal;
    float cur_color[4], cur_tex[2], cur_normal[3];
    const uint32_t *vs_ids;
    uint32_t vs_base;
    uint32_t raster;
    uint32_t vslot_base, vslot_count;
    uint32_t tri_base, tri_count;
};

// The fragment stages' part of a raster state, packed for the tile kernel: a word of the
// stage enables and each stage's operands in 16-byte groups, 160 bytes in all. The
// full state spans about a kilobyte (mostly lights and materials) and scatters these fields
// over several lines; per fragment the kernel now loads the first group, and further groups
// only for the stages its enables switch on.
enum FragCtl : uint32_t {
    FC_STENCIL = 1u << 0, FC_DEPTH = 1u << 1, FC_DEPTH_WRITE = 1u << 2, FC_FLAT = 1u << 3, FC_ALPHA = 1u << 4,
    FC_AFFINE_UV = 1u << 5, FC_FOG = 1u << 6, FC_BLEND = 1u << 7, FC_DEFAULT_RANGE = 1u << 8,
    FC_MASK_ALL = 1u << 9, FC_MASK_NONE = 1u << 10, FC_TEXTURE = 1u << 11
};
// A texture level: packed RGBA8 texels, row-major (px null: a level that cannot be built).
struct __align__(16) DevMip {
    const uint32_t *px;
    int32_t w, h;
};
struct __align__(16) FragState {
    uint32_t ctl, depth_func, alpha_func, tex_env_mode;
    uint32_t stencil_func;
    int32_t stencil_ref;
    uint32_t stencil_mask, stencil_writemask;
    uint32_t stencil_fail, stencil_zfail, stencil_zpass;
    float alpha_ref;
    uint32_t blend_src, blend_dst, fog_mode;
    float fog_density;
    float fog_start, fog_end;
    uint32_t color_mask;  // bit i: channel i written
    uint32_t pad0;
    float fog_color[4];
    float tex_env_color[4];
    DevMip level[2];                       // texture: levels 0 and 1 (see DevRaster)
    int32_t wrap_s, wrap_t, min_filter, mag_filter;
    const DevMip *chain;                   // levels 2.. (MTGL_OPT_MIPMAP_CHAIN), or null
    int32_t chain_levels, pad1;            // how many (0: the reference's two levels)
};

static_assert(sizeof(FragState) == 176 && offsetof(FragState, chain) == 160 && offsetof(FragState, stencil_func) == 16 &&
                  offsetof(FragState, stencil_fail) == 32 && offsetof(FragState, blend_src) == 48 &&
                  offsetof(FragState, fog_start) == 64 && offsetof(FragState, fog_color) == 80 &&
                  offsetof(FragState, tex_env_color) == 96 && offsetof(FragState, level) == 112 &&
                  sizeof(DevMip) == 16 && offsetof(FragState, wrap_s) == 144,
              "FragState groups are read as 16-byte words");

// Raster state with the bound texture resolved to device pointers.
struct DevRaster {
    FragState fs;          // derived from rs and tex when the draw is queued
    mtgl_raster_state rs;
    const uint32_t *tex;   // level 0, or null when texturing is off
    const uint32_t *mip1;  // level 1, or null when the reference cannot build it (w or h < 2)
    int32_t tex_w, tex_h, mip_w, mip_h;
    const DevMip *chain;   // levels 2.. of a texture built under MTGL_OPT_MIPMAP_CHAIN
    int32_t chain_levels;
    int32_t default_depth_range;
    int32_t needs_eye;     // per-fragment lighting reads eye-space interpolants
    int32_t depth_rejection;  // MTGL_OPT_DEPTH_REJECTION of the context at enqueue
    uint32_t frame;           // index of the frame (framebuffer) the draw renders into
};

struct ClearOp {
    uint32_t mask;
    int32_t x0, y0, x1, y1;
    uint32_t color;
    float depth;
    uint32_t stencil;
};

struct FrameDims {
    int32_t width, height;
    int32_t tiles_x, tiles_y;
};

// One framebuffer of a pass. A single-context pass has one frame; a batch has one per
// context. Tiles of all frames are numbered consecutively: frame f owns global tiles
// [tile_base, tile_base + tiles_x * tiles_y). Its clears are clears[clear_base .. +nclears).
struct DevFrame {
    uint32_t *color;
    float *depth;
    uint8_t *stencil;
    // page-locked host buffers the tile kernel also writes (device addresses; null: none): the
    // frame's read-back goes over the link while later tiles render
    uint32_t *host_color;
    float *host_depth;
    uint8_t *host_stencil;
    FrameDims dims;
    uint32_t tile_base;
    uint32_t clear_base, nclears;
    uint32_t occlude;  // binning may drop pairs hidden behind a triangle covering their tile (k_bin.cu)
    // clears of the whole framebuffer, when the frame has no others (nclears is 0 then): the
    // buffers and the last values
    uint32_t cleared, clear_color;
    float clear_depth;
    uint32_t clear_stencil;
    uint32_t tiles_x_inv;  // (2^32 - 1) / tiles_x: see tile_row
};
// local / tiles_x: the product with tiles_x_inv is at most one too small for local < 2^31
__device__ __forceinline__ uint32_t tile_row(const DevFrame &F, uint32_t local)
{
    const uint32_t n = (uint32_t)F.dims.tiles_x, q = __umulhi(local, F.tiles_x_inv);
    return local - q * n >= n ? q + 1 : q;
}

// ------------------------------------------------------------------ scalar helpers

__device__ __forceinline__ int32_t x86_f2i(float f)
{
    return (f >= -2147483648.0f && f < 2147483648.0f) ? (int32_t)f : INT32_MIN;
}

// Exact small conversions on the FP32 adder instead of the conversion unit, which issues at
// a fraction of the FP32 rate. For 0 <= v < 2^23 the float with bits 0x4B000000 | v is
// 2^23 + v; for a float f, 2^23 + f (or 1.5 * 2^23 + f) lies in [2^23, 2^24), where floats
// are the integers, so the sum rounded toward zero (or down) is 2^23 + the integer part of
// f (or 1.5 * 2^23 + floor f), read back from the low mantissa bits.
// (float)v for 0 <= v < 2^23
__device__ __forceinline__ float small_u2f(uint32_t v) { return __int_as_float(0x4B000000 | v) - 0x1p23f; }
// (int32_t)f, truncating, for 0 <= f < 2^23
__device__ __forceinline__ int32_t small_trunc(float f) { return __float_as_int(__fadd_rz(f, 0x1p23f)) - 0x4B000000; }
// (int32_t)floorf(f), with floorf(f) in *fl, for -2^22 <= f < 2^22
__device__ __forceinline__ int32_t small_floor(float f, float *fl)
{
    const float s = __fadd_rd(f, 0x1.8p23f);
    *fl = s - 0x1.8p23f;
    return __float_as_int(s) - 0x4B400000;
}

// Two IEEE single operations in one instruction (the packed f32x2 forms): each half rounds as
// the scalar operation does. The colour stages work on four channels at a time and are bound
// by issue slots, so they use these throughout.
#define MTGL_OP2(name, ptx)                                                                               \
    __device__ __forceinline__ float2 name(float2 a, float2 b)                                            \
    {                                                                                                     \
        float2 r;                                                                                         \
        asm("{\n .reg .b64 a, b, r;\n mov.b64 a, {%2, %3};\n mov.b64 b, {%4, %5};\n " ptx             \
            " r, a, b;\n mov.b64 {%0, %1}, r;\n}"                                                       \
            : "=f"(r.x), "=f"(r.y)                                                                        \
            : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));                                                    \
        return r;                                                                                         \
    }
MTGL_OP2(add2_rz, "add.rz.f32x2")
MTGL_OP2(mul2, "mul.rn.f32x2")
#undef MTGL_OP2
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c)
{
    float2 r;
    asm("{\n .reg .b64 a, b, c, r;\n mov.b64 a, {%2, %3};\n mov.b64 b, {%4, %5};\n mov.b64 c, {%6, %7};\n "
        "fma.rn.f32x2 r, a, b, c;\n mov.b64 {%0, %1}, r;\n}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return r;
}
__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }
// Sums as fma with a factor of one or minus one, which rounds once, as the sum does. The factor
// is read from constant memory, where the assembler cannot know its value: it contracts a
// packed mul.rn followed by add.rn, or by an fma with a literal one, into a single fma (a
// rounding less) whatever -fmad says (tests/test_gpu_colour.py sees the difference).
static __constant__ float2 k_plus_one = {1.0f, 1.0f};
static __constant__ float2 k_minus_one = {-1.0f, -1.0f};
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return fma2(a, k_plus_one, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return fma2(b, k_minus_one, a); }
__device__ __forceinline__ float2 lo2(float4 v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(float4 v) { return make_float2(v.z, v.w); }
__device__ __forceinline__ float4 join(float2 a, float2 b) { return make_float4(a.x, a.y, b.x, b.y); }
__device__ __forceinline__ float4 mul4(float4 a, float4 b) { return join(mul2(lo2(a), lo2(b)), mul2(hi2(a), hi2(b))); }
__device__ __forceinline__ float4 add4(float4 a, float4 b) { return join(add2(lo2(a), lo2(b)), add2(hi2(a), hi2(b))); }
__device__ __forceinline__ float4 scale4(float4 a, float t)
{
    return join(mul2(lo2(a), both(t)), mul2(hi2(a), both(t)));
}

// x / 255.0f (graphics.h:350-357, textures.c:294-307) for x an integer in [0, 255], without a
// division: 1/255 as the sum of two floats, fma(x, hi, x * lo). The result equals the IEEE
// quotient for every byte value (checked exhaustively with exact rational arithmetic in
// tests/test_arith.py).
constexpr float kInv255Hi = 0x1.010102p-8f, kInv255Lo = -0x1.fdfdfep-33f;
__device__ __forceinline__ float over_255(float x) { return __fmaf_rn(x, kInv255Hi, x * kInv255Lo); }
__device__ __forceinline__ float2 over_255(float2 x) { return fma2(x, both(kInv255Hi), mul2(x, both(kInv255Lo))); }
__device__ __forceinline__ float u8f(uint32_t v) { return over_255(small_u2f(v)); }

// The byte v that color_to_rgba32 stores per channel (graphics.h:337-348), as the float
// 2^23 + v, whose low byte is v: clamp, times 255, truncate. The reference clamps with two
// compares, which pass a NaN through to a conversion giving INT32_MIN, whose low byte is 0;
// saturation maps a NaN to 0 first, and every other input to the same clamped value (a -0 may
// come out as +0, which truncates to the same byte).
__device__ __forceinline__ float2 byte_bits(float a, float b)
{
    return add2_rz(mul2(make_float2(__saturatef(a), __saturatef(b)), both(255.0f)), both(0x1p23f));
}

// color_to_rgba32 (graphics.h:337-348)
__device__ __forceinline__ uint32_t pack_rgba(float r, float g, float b, float a)
{
    const float2 rg = byte_bits(r, g), ba = byte_bits(b, a);
    const uint32_t lo = __byte_perm(__float_as_uint(rg.x), __float_as_uint(rg.y), 0x0040);
    const uint32_t hi = __byte_perm(__float_as_uint(ba.x), __float_as_uint(ba.y), 0x0040);
    return __byte_perm(lo, hi, 0x5410);
}

__device__ __forceinline__ float4 unpack_rgba(uint32_t p)
{
    // a byte under the exponent of 2^23: 2^23 + v
    const float2 rg = make_float2(__uint_as_float(__byte_perm(p, 0x4B000000u, 0x7440)),
                                  __uint_as_float(__byte_perm(p, 0x4B000000u, 0x7441)));
    const float2 ba = make_float2(__uint_as_float(__byte_perm(p, 0x4B000000u, 0x7442)),
                                  __uint_as_float(__byte_perm(p, 0x4B000000u, 0x7443)));
    return join(over_255(sub2(rg, both(0x1p23f))), over_255(sub2(ba, both(0x1p23f))));
}

// unpack_rgba(pack_rgba(c)): a colour through its stored bytes
__device__ __forceinline__ float4 quantize(float4 c)
{
    return join(over_255(sub2(byte_bits(c.x, c.y), both(0x1p23f))), over_255(sub2(byte_bits(c.z, c.w), both(0x1p23f))));
}

__device__ __forceinline__ float clamp01(float v) { return v < 0.0f ? 0.0f : (v > 1.0f ? 1.0f : v); }
__device__ __forceinline__ float4 clamp4(float4 c)
{
    return make_float4(clamp01(c.x), clamp01(c.y), clamp01(c.z), clamp01(c.w));
}

// color_lerp (graphics.h:293-296): a*(1-t) + b*t
__device__ __forceinline__ float4 lerp_col(float4 a, float4 b, float t)
{
    return add4(scale4(a, 1.0f - t), scale4(b, t));
}

// color_lerp_rgb (graphics.h:298-305): a + (b-a)*t, keeps a's alpha
__device__ __forceinline__ float4 lerp_rgb(float4 a, float4 b, float t)
{
    const float2 xy = add2(lo2(a), mul2(sub2(lo2(b), lo2(a)), both(t)));
    return make_float4(xy.x, xy.y, a.z + (b.z - a.z) * t, a.w);
}

__device__ __forceinline__ float3 normalize3(float x, float y, float z)
{
    float len = sqrtf(x * x + y * y + z * z);
    if (len > 0.0f) {
        float s = 1.0f / len;
        return make_float3(x * s, y * s, z * s);
    }
    return make_float3(x, y, z);
}

// mat4_mul_vec4 (graphics.h:131-138), column-major m
__device__ __forceinline__ float4 mul_m4(const float *m, float x, float y, float z, float w)
{
    return make_float4(m[0] * x + m[4] * y + m[8] * z + m[12] * w, m[1] * x + m[5] * y + m[9] * z + m[13] * w,
                       m[2] * x + m[6] * y + m[10] * z + m[14] * w, m[3] * x + m[7] * y + m[11] * z + m[15] * w);
}

__device__ __forceinline__ bool cmp_pass(uint32_t func, float a, float b)
{
    // the comparison functions are GL_NEVER + a mask of less (1), equal (2) and greater (4); an
    // unordered pair passes GL_NOTEQUAL and GL_ALWAYS, the two with less and greater
    const uint32_t r = a < b ? 1u : (a == b ? 2u : (a > b ? 4u : 8u));
    const uint32_t f = func & 7u;
    return ((f | ((f & 5u) == 5u ? 8u : 0u)) & r) != 0u;
}
static_assert(GL_LESS == GL_NEVER + 1 && GL_EQUAL == GL_NEVER + 2 && GL_LEQUAL == GL_NEVER + 3 &&
                  GL_GREATER == GL_NEVER + 4 && GL_NOTEQUAL == GL_NEVER + 5 && GL_GEQUAL == GL_NEVER + 6 &&
                  GL_ALWAYS == GL_NEVER + 7 && (GL_NEVER & 7) == 0,
              "comparison functions as masks");

// ------------------------------------------------------------------ lighting (lighting.h:53-142)

__device__ __forceinline__ float4 ld4(const float *p) { return make_float4(p[0], p[1], p[2], p[3]); }

__device__ inline float4 compute_lighting(const mtgl_lighting &L, float3 ep, float3 en, const mtgl_material &mat)
{
    // emission + ambient * global ambient, alpha from the diffuse material
    float4 r = make_float4(mat.emission[0] + mat.ambient[0] * L.model_ambient[0],
                           mat.emission[1] + mat.ambient[1] * L.model_ambient[1],
                           mat.emission[2] + mat.ambient[2] * L.model_ambient[2],
                           mat.emission[3] + mat.ambient[3] * L.model_ambient[3]);
    r.w = mat.diffuse[3];
    float3 N = en;
    if (L.normalize) N = normalize3(N.x, N.y, N.z);
    for (int i = 0; i < MTGL_MAX_LIGHTS; i++) {
        const mtgl_light &l = L.lights[i];
        if (!l.enabled) continue;
        float3 Ld;
        float att = 1.0f;
        if (l.position[3] == 0.0f) {
            Ld = make_float3(l.dir_normalized[0], l.dir_normalized[1], l.dir_normalized[2]);
        } else {
            float tx = l.position[0] - ep.x, ty = l.position[1] - ep.y, tz = l.position[2] - ep.z;
            float dist = sqrtf(tx * tx + ty * ty + tz * tz);
            if (dist < 1e-6f) dist = 1e-6f;
            float inv = 1.0f / dist;
            Ld = make_float3(tx * inv, ty * inv, tz * inv);
            float den = l.constant_attenuation + l.linear_attenuation * dist + l.quadratic_attenuation * dist * dist;
            if (den < 1e-6f) den = 1e-6f;
            att = 1.0f / den;
            if (l.spot_cutoff < 180.0f) {
                float ca = -(Ld.x * l.spot_dir_normalized[0] + Ld.y * l.spot_dir_normalized[1] +
                             Ld.z * l.spot_dir_normalized[2]);
                if (ca < l.cos_cutoff) att = 0.0f;
                else att *= powf(ca, l.spot_exponent);
            }
        }
        if (att <= 0.0f) continue;
        r.x = r.x + (mat.ambient[0] * l.ambient[0]) * att;
        r.y = r.y + (mat.ambient[1] * l.ambient[1]) * att;
        r.z = r.z + (mat.ambient[2] * l.ambient[2]) * att;
        r.w = r.w + (mat.ambient[3] * l.ambient[3]) * att;
        float ndl = N.x * Ld.x + N.y * Ld.y + N.z * Ld.z;
        if (ndl > 0.0f) {
            float k = att * ndl;
            r.x = r.x + (mat.diffuse[0] * l.diffuse[0]) * k;
            r.y = r.y + (mat.diffuse[1] * l.diffuse[1]) * k;
            r.z = r.z + (mat.diffuse[2] * l.diffuse[2]) * k;
            r.w = r.w + (mat.diffuse[3] * l.diffuse[3]) * k;
            if (mat.shininess > 0.0f) {
                float3 V = L.local_viewer ? normalize3(ep.x * -1.0f, ep.y * -1.0f, ep.z * -1.0f)
                                          : make_float3(0.0f, 0.0f, 1.0f);
                float3 Hh = normalize3(Ld.x + V.x, Ld.y + V.y, Ld.z + V.z);
                float ndh = N.x * Hh.x + N.y * Hh.y + N.z * Hh.z;
                if (ndh > 0.0f) {
                    float sp = powf(ndh, mat.shininess) * att;
                    r.x = r.x + (mat.specular[0] * l.specular[0]) * sp;
                    r.y = r.y + (mat.specular[1] * l.specular[1]) * sp;
                    r.z = r.z + (mat.specular[2] * l.specular[2]) * sp;
                    r.w = r.w + (mat.specular[3] * l.specular[3]) * sp;
                }
            }
        }
    }
    return clamp4(r);
}

// ------------------------------------------------------------------ texture sampling (textures.c:271-557)

struct TexView {
    const uint32_t *px;
    int32_t w, h;
};

// get_texel_wrapped's coordinate rule (textures.c:272-291): GL_REPEAT is ((x % n) + n) % n,
// anything else clamps to [0, n-1]. For a power-of-two n the REPEAT result is x & (n - 1)
// (the same value for every int x, negative ones included), which avoids two integer
// divisions per coordinate.
__device__ __forceinline__ int32_t wrap_coord(int32_t x, int32_t n, bool repeat)
{
    if (repeat) return (n & (n - 1)) == 0 ? (x & (n - 1)) : ((x % n) + n) % n;
    return x < 0 ? 0 : (x >= n ? n - 1 : x);
}

// wrap_coord(x + 1) from xa = wrap_coord(x): under GL_REPEAT it is (xa + 1) mod n
__device__ __forceinline__ int32_t wrap_next(int32_t xa, int32_t x, int32_t n, bool repeat)
{
    if (repeat) return xa + 1 == n ? 0 : xa + 1;
    return wrap_coord(x + 1, n, false);
}

// One axis of a bilinear sample at texel coordinate t of an n-texel axis: the two texels and the
// weight of the second.
struct TexAxis {
    int32_t a, b;
    float f;
};
static __device__ __noinline__ TexAxis tex_axis_any(float t, int32_t n, bool repeat)
{
    const int32_t i = x86_f2i(floorf(t));
    const int32_t a = wrap_coord(i, n, repeat);
    return TexAxis{a, wrap_next(a, i, n, repeat), t - (float)i};
}
// A wrapped or clamped coordinate u in [0, 1] gives t = u * n - 0.5 in [-0.5, n - 0.5], whose
// texels need a wrap only past the ends; anything else (NaN, infinities) goes the general way.
__device__ __forceinline__ TexAxis tex_axis(float t, int32_t n, float fn, bool repeat)
{
    if (!(t >= -1.0f && t < fminf(fn, 0x1p22f))) return tex_axis_any(t, n, repeat);
    float fl;
    const int32_t i = small_floor(t, &fl);  // -1 .. n - 1
    return TexAxis{i < 0 ? (repeat ? n - 1 : 0) : i, i + 1 < n ? i + 1 : (repeat ? 0 : n - 1), t - fl};
}

// texture_sample_nearest / _linear on one level, as the colour of the stored bytes
__device__ __forceinline__ float4 sample_level(const TexView &t, int32_t ws, int32_t wt, float u, float v, bool linear)
{
    const float fw = (float)t.w, fh = (float)t.h;
    float tx = u * fw - 0.5f;
    float ty = v * fh - 0.5f;
    if (linear) {
        const TexAxis x = tex_axis(tx, t.w, fw, ws == GL_REPEAT), y = tex_axis(ty, t.h, fh, wt == GL_REPEAT);
        // a level holds at most 2^32 texels: 32-bit offsets
        const uint32_t ra = (uint32_t)y.a * (uint32_t)t.w, rb = (uint32_t)y.b * (uint32_t)t.w;
        const uint32_t p00 = __ldg(t.px + (ra + x.a)), p10 = __ldg(t.px + (ra + x.b));
        const uint32_t p01 = __ldg(t.px + (rb + x.a)), p11 = __ldg(t.px + (rb + x.b));
        const float4 top = lerp_col(unpack_rgba(p00), unpack_rgba(p10), x.f);
        const float4 bot = lerp_col(unpack_rgba(p01), unpack_rgba(p11), x.f);
        return quantize(lerp_col(top, bot, y.f));
    }
    const float hx = tx + 0.5f, hy = ty + 0.5f;
    int32_t x, y;
    float fl;
    if (fabsf(hx) < 0x1p22f && fabsf(hy) < 0x1p22f) {
        x = small_floor(hx, &fl);
        y = small_floor(hy, &fl);
    } else {
        x = x86_f2i(floorf(hx));
        y = x86_f2i(floorf(hy));
    }
    if (x < 0) x = 0;
    if (x >= t.w) x = t.w - 1;
    if (y < 0) y = 0;
    if (y >= t.h) y = t.h - 1;
    return unpack_rgba(__ldg(t.px + (uint32_t)y * (uint32_t)t.w + x));
}

// (float)x86_f2i(f): the truncated value as a float (INT32_MIN outside the int range)
__device__ __forceinline__ float trunc_f2i_f(float f)
{
    const float a = fabsf(f);
    if (!(a < 0x1p22f)) return (float)x86_f2i(f);
    const float t = __fadd_rz(a, 0x1p23f) - 0x1p23f;  // trunc |f|: +0 for |f| < 1, as (float)0 is
    return f < 0.0f ? -t : t;  // a -0 here only meets u - t, where it acts as +0
}

// Level d of a texture (0: base, 1: mip1, null when it cannot be built; 2..: the chain).
__device__ __forceinline__ TexView tex_level(const FragState &S, int d)
{
    const DevMip *m = S.level + d;
    if (d > 1)
        m = reinterpret_cast<const DevMip *>(__ldg(reinterpret_cast<const unsigned long long *>(&S.chain))) + (d - 2);
    const int4 q = __ldg(reinterpret_cast<const int4 *>(m));
    const uint64_t px = (uint64_t)(uint32_t)q.x | ((uint64_t)(uint32_t)q.y << 32);
    return TexView{reinterpret_cast<const uint32_t *>(px), q.z, q.w};
}

// texture_sample_lod (textures.c:457-557) on the packed texture state, as the colour of the
// sampled bytes. The filter picks one level, or two and a weight:
// - GL_NEAREST / GL_LINEAR (and any filter at lod <= 0): the base level;
// - *_MIPMAP_NEAREST: level 1 from lod 0.5 up;
// - *_MIPMAP_LINEAR: levels 0 and 1 blended by lod; from lod 1 up level 1 alone: lerp_col(c0,
//   c1, 1) gives c1's channels exactly (c0 * 0 + c1 * 1), and their bytes are c1's again
//   (truncating ((float)b / 255) * 255 returns b for every byte).
// With a whole chain (MTGL_OPT_MIPMAP_CHAIN; no counterpart in the reference) and lod > 0:
// level floor(lod + 0.5), or levels floor(lod) and floor(lod) + 1 blended by the fraction, and
// from the top level up that level alone.
// The levels go through one copy of the filter code, in a loop: the tile kernels spill out of
// the instruction cache otherwise (no_instruction was the largest stall of a textured frame).
__device__ inline float4 sample_lod(const FragState &S, float u, float v, float lod)
{
    const int4 mode = __ldg(reinterpret_cast<const int4 *>(&S.wrap_s));  // wrap s, wrap t, min, mag filter
    const int32_t ws = mode.x, wt = mode.y;
    if (ws == GL_REPEAT) {
        u = u - trunc_f2i_f(u);
        if (u < 0) u += 1.0f;
    } else {
        if (u < 0.0f) u = 0.0f;
        if (u > 1.0f) u = 1.0f;
    }
    if (wt == GL_REPEAT) {
        v = v - trunc_f2i_f(v);
        if (v < 0) v += 1.0f;
    } else {
        if (v < 0.0f) v = 0.0f;
        if (v > 1.0f) v = 1.0f;
    }
    const int32_t filter = (lod > 0.0f) ? mode.z : mode.w;
    const bool linear = filter == GL_LINEAR || filter == GL_LINEAR_MIPMAP_NEAREST || filter == GL_LINEAR_MIPMAP_LINEAR;
    int d = 0, last = 0;
    float t = 0.0f;
    if (lod > 0.0f && filter != GL_NEAREST && filter != GL_LINEAR) {
        const int top = 1 + __ldg(&S.chain_levels);
        if (filter == GL_NEAREST_MIPMAP_NEAREST || filter == GL_LINEAR_MIPMAP_NEAREST) {
            if (top == 1) d = lod >= 0.5f ? 1 : 0;
            else d = lod >= (float)top ? top : min((int)(lod + 0.5f), top);
            last = d;
        } else {
            d = lod >= (float)top ? top : (int)lod;
            last = min(d + 1, top);
            t = lod - (float)d;
        }
    }
    float4 c = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 1
    for (int k = d; k <= last; k++) {
        const TexView view = tex_level(S, k);
        // a level 1 that cannot be built samples as white (textures.c:317, 416-419)
        const float4 s = view.px ? sample_level(view, ws, wt, u, v, linear) : make_float4(1.0f, 1.0f, 1.0f, 1.0f);
        c = k == d ? s : quantize(lerp_col(c, s, t));
    }
    return c;
}

// ------------------------------------------------------------------ fragment helpers (raster.c:343-448, 672-705)

__device__ __forceinline__ float4 blend_factor(uint32_t f, float4 s, float4 d)
{
    switch (f) {
    case GL_ZERO: return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    case GL_ONE: return make_float4(1.0f, 1.0f, 1.0f, 1.0f);
    case GL_SRC_COLOR: return s;
    case GL_ONE_MINUS_SRC_COLOR: return make_float4(1 - s.x, 1 - s.y, 1 - s.z, 1 - s.w);
    case GL_DST_COLOR: return d;
    case GL_ONE_MINUS_DST_COLOR: return make_float4(1 - d.x, 1 - d.y, 1 - d.z, 1 - d.w);
    case GL_SRC_ALPHA: return make_float4(s.w, s.w, s.w, s.w);
    case GL_ONE_MINUS_SRC_ALPHA: { float k = 1 - s.w; return make_float4(k, k, k, k); }
    case GL_DST_ALPHA: return make_float4(d.w, d.w, d.w, d.w);
    case GL_ONE_MINUS_DST_ALPHA: { float k = 1 - d.w; return make_float4(k, k, k, k); }
    case GL_SRC_ALPHA_SATURATE: {
        float k = (s.w < (1 - d.w)) ? s.w : (1 - d.w);
        return make_float4(k, k, k, 1.0f);
    }
    default: return make_float4(1.0f, 1.0f, 1.0f, 1.0f);
    }
}

// The result is clamped where it is stored (pack_rgba): the reference's clamp before that
// changes nothing, and a masked write keeps the same channels.
__device__ __forceinline__ float4 blend(uint32_t src, uint32_t dst, float4 s, float4 d)
{
    if (src == GL_SRC_ALPHA && dst == GL_ONE_MINUS_SRC_ALPHA)  // the common pair, without the two switches
        return add4(scale4(s, s.w), scale4(d, 1 - s.w));
    return add4(mul4(s, blend_factor(src, s, d)), mul4(d, blend_factor(dst, s, d)));
}

__device__ __forceinline__ float4 blend(const mtgl_raster_state &rs, float4 s, float4 d)
{
    return blend(rs.blend_src, rs.blend_dst, s, d);
}

__device__ __forceinline__ bool stencil_pass(uint32_t func, int32_t ref, uint32_t mask, uint32_t val)
{
    const int32_t mr = (int32_t)((uint32_t)ref & mask);
    const int32_t mv = (int32_t)(val & mask);
    return (func & (mr < mv ? 1u : (mr == mv ? 2u : 4u))) != 0u;  // see cmp_pass
}

__device__ __forceinline__ uint32_t stencil_apply(uint32_t op, uint32_t v, int32_t ref)
{
    switch (op) {
    case GL_KEEP: return v;
    case GL_ZERO: return 0u;
    case GL_REPLACE: return (uint32_t)ref & 0xFFu;
    case GL_INCR: return v < 255u ? v + 1u : 255u;
    case GL_INCR_WRAP: return (v + 1u) & 0xFFu;
    case GL_DECR: return v > 0u ? v - 1u : 0u;
    case GL_DECR_WRAP: return (v - 1u) & 0xFFu;
    case GL_INVERT: return (~v) & 0xFFu;
    default: return v;
    }
}

__device__ __forceinline__ uint32_t stencil_write(uint32_t old, uint32_t nv, uint32_t writemask)
{
    uint32_t m8 = writemask & 0xFFu;
    return ((old & ~m8) | (nv & m8)) & 0xFFu;
}

__device__ __forceinline__ float fog_factor(uint32_t mode, float density, float start, float end, float fog_coord)
{
    float f;
    switch (mode) {
    case GL_LINEAR:
        f = (end != start) ? (end - fog_coord) / (end - start) : 1.0f;
        break;
    case GL_EXP: f = expf(-density * fog_coord); break;
    case GL_EXP2: {
        float d = density * fog_coord;
        f = expf(-d * d);
        break;
    }
    default: f = 1.0f; break;
    }
    if (f < 0.0f) f = 0.0f;
    if (f > 1.0f) f = 1.0f;
    return f;
}

__device__ __forceinline__ float fog_factor(const mtgl_raster_state &rs, float fog_coord)
{
    return fog_factor(rs.fog_mode, rs.fog_density, rs.fog_start, rs.fog_end, fog_coord);
}

// the double-precision depth range map, out of line: inlined, its few FP64 instructions
// are issued (predicated off) for every fragment of the default range as well, and the
// FP64 pipe of this GPU is narrow
static __device__ __noinline__ float map_depth_range(float t, double near_d, double far_d)
{
    return (float)((double)t * (far_d - near_d) + near_d);
}

// depth range mapping (raster.c:548): float NDC term, double range, float result
__device__ __forceinline__ float map_depth(const DevRaster &R, float z)
{
    float t = (z + 1.0f) * 0.5f;
    if (R.default_depth_range) return t;  // (double)t * 1.0 + 0.0 rounds back to t
    return map_depth_range(t, R.rs.depth_near, R.rs.depth_far);
}

// write_pixel_masked (raster.c:20-45) on a packed destination pixel; mask bit i: channel i
__device__ __forceinline__ uint32_t masked_write(uint32_t mask, uint32_t dst, float4 c)
{
    if (mask == 15u) return pack_rgba(c.x, c.y, c.z, c.w);
    if (mask == 0u) return dst;
    float4 d = unpack_rgba(dst);
    if (mask & 1u) d.x = c.x;
    if (mask & 2u) d.y = c.y;
    if (mask & 4u) d.z = c.z;
    if (mask & 8u) d.w = c.w;
    return pack_rgba(d.x, d.y, d.z, d.w);
}

__device__ __forceinline__ uint32_t masked_write(const mtgl_raster_state &rs, uint32_t dst, float4 c)
{
    const uint32_t *m = rs.color_mask;
    return masked_write((m[0] ? 1u : 0u) | (m[1] ? 2u : 0u) | (m[2] ? 4u : 0u) | (m[3] ? 8u : 0u), dst, c);
}

}  // namespace mtgl
