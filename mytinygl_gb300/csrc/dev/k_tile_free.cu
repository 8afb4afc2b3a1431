// k_tile_free.cu — K4 for order-free passes (raster.c:532-724, gl_api.c:409-457).
//
// In a pass whose every record is a filled triangle that tests and writes depth with GL_LESS
// (or GL_LEQUAL, one function per frame), has no stencil test, blending or discards and writes
// all four channels, a pixel ends with the depth and colour of its nearest fragment: of equal
// depths the first in submission order under GL_LESS, the last under GL_LEQUAL. That is the
// smallest (depth, record index) pair (or the largest index), whatever order the fragments are
// taken in, so binning neither sorts nor orders the tile lists, records may be skipped on any
// sound bound, and the colour stages run once per pixel.
//
// One CTA per tile, one thread per pixel, one warp per 8x4 block. The tile's records are staged
// 64 at a time into shared memory with asynchronous copies, the next chunk in flight while one
// is walked: the walk itself then reads no global memory. Each warp tests 32 staged records at
// once, a lane each, against its block: whether any pixel can be covered, whether all are, and
// the record's smallest and largest depth there; the nearest of the largest depths over
// records that cover the whole block bounds every other record. What is left is taken record
// by record (all lanes evaluate one triangle) when it is little, else by coverage masks: each
// lane finds its record's 32-bit mask over the block's pixels, the masks are transposed across
// the warp, and every lane takes the records of its own pixel one per round.
//
// What bounds it: latency of the chain list -> records -> colour operands -> texels per tile,
// hidden by the resident CTAs, and issue of the colour stages.
#include "k_tile.cuh"

namespace mtgl {

namespace {

constexpr int kStage = 64;         // records staged at a time
constexpr int kStageWords = 9;     // 16-byte words per staged record: 7 used, stride free of bank conflicts
// record words in stage order: q0 q1 q2 q3 q12 q13 q14, then the record index
enum StageWord { SW_Q0, SW_Q1, SW_Q2, SW_Q3, SW_Q12, SW_Q13, SW_Q14, SW_INDEX };
constexpr int kPerRecordMax = 6;   // records of a step taken one by one; more go by masks

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem)
{
    const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// 32x32 bit transpose across the warp: bit i of lane l becomes bit l of lane i.
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

struct Nearest {
    float dep;     // the pixel's depth
    uint32_t rec;  // 1 + the record that holds it, 0: none
};

// One fragment: the reference's depth at the pixel, kept when it is the nearer.
__device__ __forceinline__ bool take_fragment(const TileArgs &A, const float4 *q, float fpx, float fpy, Nearest &n)
{
    const float4 q0 = q[SW_Q0], q1 = q[SW_Q1], q2 = q[SW_Q2], q3 = q[SW_Q3], q12 = q[SW_Q12], q13 = q[SW_Q13];
    const float e0 = (fpx - q0.z) * q12.y - (fpy - q0.w) * q12.z;
    const float e1 = (fpx - q1.x) * q12.w - (fpy - q1.y) * q13.x;
    const float e2 = (fpx - q0.x) * q13.y - (fpy - q0.y) * q13.z;
    const float b0 = e0 * q2.w, b1 = e1 * q2.w, b2 = e2 * q2.w;
    const float z = b0 * q3.x + b1 * q3.y + b2 * q3.z;
    float depth = (z + 1.0f) * 0.5f;
    const uint32_t flags = __float_as_uint(q12.x), idx = __float_as_uint(q[SW_INDEX].x);
    if (!((flags >> kRecCtlShift) & FC_DEFAULT_RANGE)) {
        const uint32_t rs = __float_as_uint(__ldg(A.records + (size_t)idx * kRecWords + R_RASTER));
        const DevRaster &R = A.rasters[min(rs, A.nrasters - 1)];
        depth = map_depth_range(depth, R.rs.depth_near, R.rs.depth_far);
    }
    const bool less = ((flags >> kRecDepthFuncShift) & 7u) == GL_LESS - GL_NEVER;
    const bool tie = less ? idx + 1u < n.rec : idx + 1u > n.rec;
    const bool pass = depth < n.dep || (depth == n.dep && tie);
    if (pass) {
        n.dep = depth;
        n.rec = idx + 1u;
    }
    return pass;
}

// the coverage test of rasterize_triangle_smooth at the pixel (raster.c:534-540), box included
__device__ __forceinline__ bool covers(const float4 *q, int px, int py, float fpx, float fpy)
{
    const float4 q0 = q[SW_Q0], q1 = q[SW_Q1], q2 = q[SW_Q2], q12 = q[SW_Q12], q13 = q[SW_Q13];
    if (px < __float_as_int(q1.z) || px > __float_as_int(q2.x) || py < __float_as_int(q1.w) ||
        py > __float_as_int(q2.y))
        return false;
    const float e0 = (fpx - q0.z) * q12.y - (fpy - q0.w) * q12.z;
    const float e1 = (fpx - q1.x) * q12.w - (fpy - q1.y) * q13.x;
    const float e2 = (fpx - q0.x) * q13.y - (fpy - q0.y) * q13.z;
    return (q2.z > 0 && e0 >= 0 && e1 >= 0 && e2 >= 0) || (q2.z < 0 && e0 <= 0 && e1 <= 0 && e2 <= 0);
}

// A staged record against the warp's block. The per-pixel test of edge k is p >= r with p =
// (x - ax) * A and r = (y - ay) * B as floats (a difference of floats has the sign of their
// order), both sides negated for a negative area; p is monotone in x and r in y, rounding
// included, so their extremes over the block's part of the box are at its corners, exactly.
struct BlockTest {
    bool any, all;  // some pixel may be covered / every pixel of the block in the framebuffer is
    float lo, hi;   // bounds of the record's depths there (-inf, +inf without one)
};
__device__ __forceinline__ BlockTest test_block(const float4 *q, int wx0, int wy0, int wx1, int wy1)
{
    const float4 q0 = q[SW_Q0], q1 = q[SW_Q1], q2 = q[SW_Q2], q12 = q[SW_Q12], q13 = q[SW_Q13];
    const int mnx = __float_as_int(q1.z), mny = __float_as_int(q1.w);
    const int xl = max(wx0, mnx), xh = min(wx1, __float_as_int(q2.x));
    const int yl = max(wy0, mny), yh = min(wy1, __float_as_int(q2.y));
    BlockTest t;
    const float sg = q2.z > 0.0f ? 1.0f : -1.0f;
    t.any = xl <= xh && yl <= yh && (q2.z > 0.0f || q2.z < 0.0f);
    t.all = t.any && xl == wx0 && xh == wx1 && yl == wy0 && yh == wy1;
    const float fxl = (float)xl, fxh = (float)xh, fyl = (float)yl, fyh = (float)yh;
    const float ax[3] = {q0.z, q1.x, q0.x}, ay[3] = {q0.w, q1.y, q0.y};
    const float ea[3] = {q12.y, q12.w, q13.y}, eb[3] = {q12.z, q13.x, q13.z};
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const float a = ea[k] * sg, b = eb[k] * sg;
        const float p0 = (fxl - ax[k]) * a, p1 = (fxh - ax[k]) * a;
        const float r0 = (fyl - ay[k]) * b, r1 = (fyh - ay[k]) * b;
        t.any = t.any && fmaxf(p0, p1) >= fminf(r0, r1);
        t.all = t.all && fminf(p0, p1) >= fmaxf(r0, r1);
    }
    t.lo = -INFINITY;
    t.hi = INFINITY;
    const uint32_t zc = (__float_as_uint(q12.x) >> 1) & 3u;
    if (t.any && (zc == ZC_LESS || zc == ZC_LEQUAL)) {
        const float4 zp = q[SW_Q14];
        t.lo = fmaxf(q[SW_Q3].w, depth_plane_bound(zp, mnx, mny, xl, xh, yl, yh));
        if (t.all && isfinite(zp.w)) t.hi = depth_plane_upper(zp, mnx, mny, xl, xh, yl, yh);
    }
    return t;
}

// The record's covered pixels of the block at (wx0, wy0), bit 8 * row + column: the per-pixel
// test in the form above.
__device__ __forceinline__ uint32_t cover_mask(const float4 *q, int wx0, int wy0)
{
    const float4 q0 = q[SW_Q0], q1 = q[SW_Q1], q2 = q[SW_Q2], q12 = q[SW_Q12], q13 = q[SW_Q13];
    const float sg = q2.z > 0.0f ? 1.0f : -1.0f;
    const float ax[3] = {q0.z, q1.x, q0.x}, ay[3] = {q0.w, q1.y, q0.y};
    const float ea[3] = {q12.y, q12.w, q13.y}, eb[3] = {q12.z, q13.x, q13.z};
    float p[3][8];
#pragma unroll
    for (int k = 0; k < 3; k++)
#pragma unroll
        for (int c = 0; c < 8; c++) p[k][c] = ((float)(wx0 + c) - ax[k]) * (ea[k] * sg);
    const int c0 = max(__float_as_int(q1.z) - wx0, 0), c1 = min(__float_as_int(q2.x) - wx0, 7);
    const uint32_t cols = c0 <= c1 ? (0xFFu >> (7 - c1)) & (0xFFu << c0) : 0u;
    const int r0 = __float_as_int(q1.w) - wy0, r1 = __float_as_int(q2.y) - wy0;
    uint32_t m = 0;
#pragma unroll
    for (int r = 0; r < 4; r++) {
        float y[3];
#pragma unroll
        for (int k = 0; k < 3; k++) y[k] = ((float)(wy0 + r) - ay[k]) * (eb[k] * sg);
        uint32_t bits = 0;
#pragma unroll
        for (int c = 0; c < 8; c++)
            if (p[0][c] >= y[0] && p[1][c] >= y[1] && p[2][c] >= y[2]) bits |= 1u << c;
        if (r >= r0 && r <= r1) m |= (bits & cols) << (8 * r);
    }
    return m;
}

template <int TS>
constexpr int free_min_blocks()
{
    return TS == 32 ? 1 : 1280 / (TS * TS);
}

template <int TS, bool TEX, bool EYE>
__global__ void __launch_bounds__(TS *TS, free_min_blocks<TS>()) k_tile_free(TileArgs A)
{
    constexpr int kWarpsX = TS / 8, kThreads = TS * TS;
    __shared__ float4 s_rec[2][kStage * kStageWords];

    if (A.guard && (A.guard[0] > A.records_cap || A.guard[1] > A.pairs_cap)) return;
    const uint32_t tile = A.order ? A.order[blockIdx.x] : blockIdx.x;
    const uint32_t count = A.tile_count[tile], start = A.tile_start[tile] - count;  // tile_start: the list's end
    const DevFrame &F = A.frames[A.tile_frame ? A.tile_frame[tile] : 0u];
    const ClearOp *clears = A.clears + F.clear_base;
    const int nclears = (int)F.nclears;
    if (count == 0 && nclears == 0) return;
    if (!debug_check(A.debug, (uint64_t)start + count <= A.entries_cap, DBG_TILE_ENTRY)) return;

    // stage records [base, base + kStage) of the list: four threads per record
    auto stage = [&](uint32_t base, int buf) {
        const uint32_t m = min((uint32_t)kStage, count - base);
        for (uint32_t i = threadIdx.x; i < 4 * m; i += kThreads) {
            const uint32_t e = i >> 2, part = i & 3u;
            uint32_t idx = __ldg(A.tile_vals + start + base + e);
            if (!debug_check(A.debug, idx < A.records_cap, DBG_TILE_RECORD)) idx = 0;
            const float4 *q = reinterpret_cast<const float4 *>(A.records + (size_t)idx * kRecWords);
            float4 *d = s_rec[buf] + e * kStageWords;
            const uint32_t from = part < 2 ? 2 * part : 8 + 2 * part;  // words 0 1 | 2 3 | 12 13 | 14
            cp_async16(d + 2 * part, q + from);
            if (part < 3) cp_async16(d + 2 * part + 1, q + from + 1);
            else d[SW_INDEX].x = __uint_as_float(idx);
        }
    };
    if (count) stage(0, 0);
    cp_async_commit();

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t local = tile - F.tile_base;
    const int tx = (int)(local % (uint32_t)F.dims.tiles_x), ty = (int)(local / (uint32_t)F.dims.tiles_x);
    const int W = F.dims.width, H = F.dims.height;
    const int wx0 = tx * TS + (warp % kWarpsX) * 8, wy0 = ty * TS + (warp / kWarpsX) * 4;
    const int wx1 = min(wx0 + 7, W - 1), wy1 = min(wy0 + 3, H - 1);  // the block's part of the framebuffer
    const int px = wx0 + (lane & 7), py = wy0 + (lane >> 3);
    const bool in_fb = px < W && py < H;
    const size_t pix = (size_t)py * W + px;

    // the clears; buffers a clear fully covers are never loaded, and the stencil buffer is
    // touched by clears alone
    const int bx0 = tx * TS, by0 = ty * TS, bx1 = min(bx0 + TS, W), by1 = min(by0 + TS, H);
    bool load_c = true, load_d = true, load_s = false;
    uint32_t cleared = 0;
    for (int i = 0; i < nclears; i++) {
        const ClearOp &c = clears[i];
        if (covers_tile(c, GL_COLOR_BUFFER_BIT, bx0, by0, bx1, by1)) load_c = false;
        if (covers_tile(c, GL_DEPTH_BUFFER_BIT, bx0, by0, bx1, by1)) load_d = false;
        if (covers_tile(c, GL_STENCIL_BUFFER_BIT, bx0, by0, bx1, by1)) load_s = false;
        else if (c.mask & GL_STENCIL_BUFFER_BIT) load_s = true;
        cleared |= c.mask;
    }
    const bool stencil = (cleared & GL_STENCIL_BUFFER_BIT) != 0;
    uint32_t col = 0, st = 0;
    Nearest n{1.0f, 0u};
    if (in_fb) {
        if (load_c) col = F.color[pix];
        if (load_d) n.dep = F.depth[pix];
        if (load_s) st = F.stencil[pix];
        for (int i = 0; i < nclears; i++) {
            const ClearOp &c = clears[i];
            if (px >= c.x0 && px < c.x1 && py >= c.y0 && py < c.y1) {
                if (c.mask & GL_COLOR_BUFFER_BIT) col = c.color;
                if (c.mask & GL_DEPTH_BUFFER_BIT) n.dep = c.depth;
                if (c.mask & GL_STENCIL_BUFFER_BIT) st = c.stencil & 0xFFu;
            }
        }
    }

    const float fpx = (float)px, fpy = (float)py;
    // no fragment beyond this depth changes a pixel of the block: the largest stored depth, or
    // the largest depth of a record of the list that covers the block
    float far = warp_max_depth(n.dep, in_fb);
    uint32_t frags = 0;
    int buf = 0;
    for (uint32_t base = 0; base < count; base += kStage, buf ^= 1) {
        cp_async_wait_all();
        __syncthreads();
        if (base + kStage < count) {
            stage(base + kStage, buf ^ 1);
            cp_async_commit();
        }
        if (wx0 >= W || wy0 >= H) continue;  // the block lies outside the framebuffer
        const int m = (int)min((uint32_t)kStage, count - base);
        for (int s0 = 0; s0 < m; s0 += 32) {
            const float4 *rec = s_rec[buf] + s0 * kStageWords;
            BlockTest t{false, false, -INFINITY, INFINITY};
            if (s0 + lane < m) t = test_block(rec + lane * kStageWords, wx0, wy0, wx1, wy1);
            if (__any_sync(0xffffffffu, t.all))
                far = fminf(far, ordered_float(__reduce_min_sync(0xffffffffu, ordered_key(t.hi))));
            uint32_t todo = __ballot_sync(0xffffffffu, t.any && !(t.lo > far));
            if (__popc(todo) <= kPerRecordMax) {
                for (; todo; todo &= todo - 1) {
                    const int j = __ffs(todo) - 1;
                    if (__shfl_sync(0xffffffffu, t.lo, j) > far) continue;
                    const float4 *q = rec + j * kStageWords;
                    bool wrote = false;
                    if (covers(q, px, py, fpx, fpy)) {
                        frags++;
                        wrote = take_fragment(A, q, fpx, fpy, n);
                    }
                    if (__any_sync(0xffffffffu, wrote)) far = fminf(far, warp_max_depth(n.dep, in_fb));
                }
            } else {
                uint32_t cov = 0;
                if ((todo >> lane) & 1u) cov = cover_mask(rec + lane * kStageWords, wx0, wy0);
                cov = warp_transpose(cov);
                frags += __popc(cov);
                while (__any_sync(0xffffffffu, cov != 0)) {
                    if (cov) {
                        take_fragment(A, rec + (__ffs(cov) - 1) * kStageWords, fpx, fpy, n);
                        cov &= cov - 1;
                    }
                }
                far = fminf(far, warp_max_depth(n.dep, in_fb));
            }
        }
    }

    if (n.rec) col = pending_color<TEX, EYE>(A, n.rec - 1u, EYE && A.eye_records != nullptr, fpx, fpy);
    if (in_fb && debug_check(A.debug, pix < (size_t)W * (size_t)H, DBG_TILE_PIXEL)) {
        F.color[pix] = col;
        F.depth[pix] = n.dep;
        if (stencil) F.stencil[pix] = (uint8_t)st;
    }
    if (A.fragments) {
        const uint32_t fw = __reduce_add_sync(0xffffffffu, frags);
        if (lane == 0 && fw) atomicAdd(A.fragments, (unsigned long long)fw);
    }
}

template <int TS>
void launch_free(const TileArgs &a, cudaStream_t s)
{
    if (a.any_texture && a.eye_records) k_tile_free<TS, true, true><<<a.ntiles, TS * TS, 0, s>>>(a);
    else if (a.any_texture) k_tile_free<TS, true, false><<<a.ntiles, TS * TS, 0, s>>>(a);
    else if (a.eye_records) k_tile_free<TS, false, true><<<a.ntiles, TS * TS, 0, s>>>(a);
    else k_tile_free<TS, false, false><<<a.ntiles, TS * TS, 0, s>>>(a);
}

}  // namespace

int launch_tile_free(const TileArgs &a, cudaStream_t s)
{
    if (a.ntiles == 0) return 0;
    switch (a.tile_shift) {
    case 3: launch_free<8>(a, s); break;
    case 5: launch_free<32>(a, s); break;
    default: launch_free<16>(a, s); break;
    }
    return 1;
}

}  // namespace mtgl
