// k_tile_free.cu — K4 for order-free passes (raster.c:532-724, gl_api.c:409-457).
//
// In a pass whose every record is a filled triangle that tests and writes depth with GL_LESS
// (or GL_LEQUAL, one function per frame), has no stencil test, blending or discards and writes
// all four channels, a pixel ends with the depth and colour of its nearest fragment: of equal
// depths the first in submission order under GL_LESS, the last under GL_LEQUAL. That is the
// smallest (depth, place) pair (or the largest place), whatever order the fragments are taken
// in, so set-up and binning order nothing, records may be skipped on any sound bound, and the
// colour stages run once per pixel. Frames without a depth test (or with GL_ALWAYS) end with
// the last fragment: the largest place alone.
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
enum StageWord { SW_Q0, SW_Q1, SW_Q2, SW_Q3, SW_Q12, SW_Q13, SW_Q14, SW_INDEX };  // SW_INDEX: index, place + 1
constexpr int kPerRecordMax = 6;   // records of a step taken one by one; more go by masks

struct Nearest {
    float dep;     // the pixel's depth
    uint32_t rec;  // the record that holds it
    uint32_t seq;  // 1 + its place in the submission order, 0: none holds it
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
    const uint32_t seq = __float_as_uint(q[SW_INDEX].y), ctl = flags >> kRecCtlShift;
    if (!(ctl & FC_DEFAULT_RANGE)) {
        const uint32_t rs = __float_as_uint(__ldg(A.records + (size_t)idx * kRecWords + R_RASTER));
        const DevRaster &R = A.rasters[min(rs, A.nrasters - 1)];
        depth = map_depth_range(depth, R.rs.depth_near, R.rs.depth_far);
    }
    const uint32_t func = (flags >> kRecDepthFuncShift) & 7u;  // a mask, see cmp_pass
    const bool later = seq > n.seq;
    bool pass = later;  // no depth test, or one that always passes
    if ((ctl & FC_DEPTH) && func != 7u)
        pass = depth < n.dep || (depth == n.dep && (func == 1u ? seq < n.seq : later));
    if (pass) {
        if (ctl & FC_DEPTH_WRITE) n.dep = depth;
        n.rec = idx;
        n.seq = seq;
    }
    return pass;
}

__device__ __forceinline__ EdgeWords edges_of(const float4 *q)
{
    return EdgeWords{q[SW_Q0], q[SW_Q1], q[SW_Q2], q[SW_Q12], q[SW_Q13]};
}

// A staged record against the warp's block, [wx0, wx1] x [wy0, wy1] in the framebuffer.
struct BlockTest {
    bool any, all;  // some pixel may be covered / every one is
    float lo, hi;   // bounds of the record's depths there (-inf, +inf without one)
};
__device__ __forceinline__ BlockTest test_block(const float4 *q, int wx0, int wy0, int wx1, int wy1)
{
    const EdgeWords w = edges_of(q);
    const int mnx = __float_as_int(w.q1.z), mny = __float_as_int(w.q1.w);
    const int xl = max(wx0, mnx), xh = min(wx1, __float_as_int(w.q2.x));
    const int yl = max(wy0, mny), yh = min(wy1, __float_as_int(w.q2.y));
    BlockTest t{false, false, -INFINITY, INFINITY};
    if (xl > xh || yl > yh) return t;
    corner_test(w, xl, xh, yl, yh, t.any, t.all);
    t.all = t.all && xl == wx0 && xh == wx1 && yl == wy0 && yh == wy1;
    const uint32_t zc = (__float_as_uint(w.q12.x) >> 1) & 3u;
    if (t.any && (zc == ZC_LESS || zc == ZC_LEQUAL)) {
        const float4 zp = q[SW_Q14];
        t.lo = fmaxf(q[SW_Q3].w, depth_plane_bound(zp, mnx, mny, xl, xh, yl, yh));
        if (t.all && isfinite(zp.w)) t.hi = depth_plane_upper(zp, mnx, mny, xl, xh, yl, yh);
    }
    return t;
}

template <int TS>
constexpr int free_min_blocks()
{
    return TS == 32 ? 1 : 1024 / (TS * TS);
}

template <int TS, bool TEX, bool EYE>
__global__ void __launch_bounds__(TS *TS, free_min_blocks<TS>()) k_tile_free(TileArgs A)
{
    constexpr int kThreads = TS * TS;
    __shared__ float4 s_rec[2][kStage * kStageWords];
    __shared__ HostTile<TS> s_out;

    const bool over = over_capacity(A);  // waited for with the first tile's words
    const int lane = threadIdx.x & 31;
    uint32_t frags = 0;
    for (uint32_t it = blockIdx.x; it < A.ntiles; it += gridDim.x) {
        const uint32_t tile = A.order ? A.order[it] : it;
        const uint32_t count = A.tile_count[tile], start = A.tile_start[tile];
        const DevFrame &F = A.frames[A.tile_frame ? A.tile_frame[tile] : 0u];
        if (over) return;
        if (idle_tile(F, count)) continue;
        if (!debug_check(A.debug, (uint64_t)start + count <= A.entries_cap, DBG_TILE_ENTRY)) continue;
        if (it != blockIdx.x) __syncthreads();  // the previous tile's records are done with

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
                else
                    *reinterpret_cast<uint2 *>(d + SW_INDEX) =
                        make_uint2(idx, (A.rec_seq ? __ldg(A.rec_seq + idx) : idx) + 1u);
            }
        };
        if (count) stage(0, 0);
        cp_async_commit();

        const TilePixel t = open_tile<TS>(A, F, tile, false);
        Nearest n{t.dep, 0u, 0u};
        uint32_t col = t.col;
        const float fpx = (float)t.px(), fpy = (float)t.py();
        // no fragment beyond this depth changes a pixel of the block: the largest stored depth, or
        // the largest depth of a record of the list that covers the block
        float far = warp_max_depth(n.dep, t.in_fb());
        int buf = 0;
        for (uint32_t base = 0; base < count; base += kStage, buf ^= 1) {
            cp_async_wait_all();
            __syncthreads();
            if (base + kStage < count) {
                stage(base + kStage, buf ^ 1);
                cp_async_commit();
            }
            if (t.wx1 < t.wx0 || t.wy1 < t.wy0) continue;  // the block lies outside the framebuffer
            const int m = (int)min((uint32_t)kStage, count - base);
            for (int s0 = 0; s0 < m; s0 += 32) {
                const float4 *rec = s_rec[buf] + s0 * kStageWords;
                BlockTest b{false, false, -INFINITY, INFINITY};
                if (s0 + lane < m) b = test_block(rec + lane * kStageWords, t.wx0, t.wy0, t.wx1, t.wy1);
                if (__any_sync(0xffffffffu, b.all))
                    far = fminf(far, ordered_float(__reduce_min_sync(0xffffffffu, ordered_key(b.hi))));
                uint32_t todo = __ballot_sync(0xffffffffu, b.any && !(b.lo > far));
                if (__popc(todo) <= kPerRecordMax) {
                    for (; todo; todo &= todo - 1) {
                        const int j = __ffs(todo) - 1;
                        if (__shfl_sync(0xffffffffu, b.lo, j) > far) continue;
                        const float4 *q = rec + j * kStageWords;
                        bool wrote = false;
                        const EdgeWords w = edges_of(q);
                        if (box_holds(w, t.px(), t.py()) && tri_covers(w, fpx, fpy)) {
                            frags++;
                            wrote = take_fragment(A, q, fpx, fpy, n);
                        }
                        if (__any_sync(0xffffffffu, wrote)) far = fminf(far, warp_max_depth(n.dep, t.in_fb()));
                    }
                } else {
                    uint32_t cov = 0;
                    if ((todo >> lane) & 1u) {
                        const EdgeWords w = edges_of(rec + lane * kStageWords);
                        cov = box_mask(w, t.wx0, t.wy0) & tri_mask(w, t.wx0, t.wy0);
                    }
                    cov = warp_transpose(cov);
                    frags += __popc(cov);
                    while (__any_sync(0xffffffffu, cov != 0)) {
                        if (cov) {
                            take_fragment(A, rec + (__ffs(cov) - 1) * kStageWords, fpx, fpy, n);
                            cov &= cov - 1;
                        }
                    }
                    far = fminf(far, warp_max_depth(n.dep, t.in_fb()));
                }
            }
        }
        if (n.seq) col = pending_color<TEX, EYE>(A, n.rec, EYE && A.eye_records != nullptr, fpx, fpy);
        close_tile<TS>(A, F, t, col, n.dep, t.st, &s_out);
    }
    if (A.fragments) {
        const uint32_t fw = __reduce_add_sync(0xffffffffu, frags);
        if (lane == 0 && fw) atomicAdd(A.fragments, (unsigned long long)fw);
    }
}

template <class Fn>
auto with_free_kernel(const TileArgs &a, Fn fn)
{
    const bool eye = a.eye_records != nullptr;
    auto pick = [&](auto none, auto tex, auto eyes, auto both_, int threads) {
        return fn(a.any_texture ? (eye ? both_ : tex) : (eye ? eyes : none), threads);
    };
    switch (a.tile_shift) {
    case 3: return pick(k_tile_free<8, false, false>, k_tile_free<8, true, false>, k_tile_free<8, false, true>, k_tile_free<8, true, true>, 64);
    case 5: return pick(k_tile_free<32, false, false>, k_tile_free<32, true, false>, k_tile_free<32, false, true>, k_tile_free<32, true, true>, 1024);
    default: return pick(k_tile_free<16, false, false>, k_tile_free<16, true, false>, k_tile_free<16, false, true>, k_tile_free<16, true, true>, 256);
    }
}

}  // namespace

int launch_tile_free(const TileArgs &a, cudaStream_t s)
{
    with_free_kernel(a, [&](auto k, int threads) { launch_tiles(k, a, threads, s); });
    return 1;
}

int free_per_sm(const TileArgs &a)
{
    return with_free_kernel(a, [](auto k, int threads) { return tiles_per_sm(k, threads); });
}

}  // namespace mtgl
