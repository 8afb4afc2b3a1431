// k_bin.cu — K3 binning: triangle records -> per-tile lists in submission order.
//
// No counterpart in the reference, which scans every triangle's bounding box on one thread
// (raster.c:532-724). Here each record is expanded into one (tile, record) pair per tile
// (8, 16 or 32 pixels square) of its clamped bounding box in which it can cover a pixel (an
// exact edge test per tile for triangles) and is not hidden there by a triangle that covers
// the whole tile. Pairs are generated in submission order and a stable LSD radix sort on the
// tile id (warp match-any ranking plus prefix sums) groups them by tile while keeping that
// order inside every tile. The tile kernel then walks each list front to back, so blending
// and stencil updates happen in GL order. Passes whose result does not depend on that order
// (k_tile_free.cu) skip the sort: their pairs go straight to the tiles' lists.
#include <algorithm>

#include "dev_kernels.h"

namespace mtgl {

// ------------------------------------------------------------------ scan

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;  // 2048 values per block

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v)
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t n = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += n;
    }
    return v;
}

// Sums that stay at the largest value instead of wrapping, so that a total past 32 bits is seen as
// one that fits nowhere. (Saturating addition of unsigned numbers is associative: the sum, or
// the limit.) Scans whose total decides nothing (SAT false) add plainly.
template <bool SAT>
__device__ __forceinline__ uint32_t add_to(uint32_t a, uint32_t b)
{
    const uint32_t s = a + b;
    return SAT && s < a ? 0xFFFFFFFFu : s;
}
// scan over the warp: returns the exclusive sum, the inclusive one in *incl
template <bool SAT>
__device__ __forceinline__ uint32_t warp_excl_scan(uint32_t v, uint32_t *incl)
{
    const int lane = threadIdx.x & 31;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t n = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x = add_to<SAT>(x, n);
    }
    *incl = x;
    if (!SAT) return x - v;
    const uint32_t before = __shfl_up_sync(0xffffffffu, x, 1);
    return lane ? before : 0u;
}

// exclusive block scan of one value per thread; returns the block total in *total
template <bool SAT>
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t *total)
{
    __shared__ uint32_t warp_sums[kScanThreads / 32 + 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl;
    const uint32_t before = warp_excl_scan<SAT>(v, &incl);
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        uint32_t wi;
        const uint32_t wb = warp_excl_scan<SAT>(lane < kScanThreads / 32 ? warp_sums[lane] : 0u, &wi);
        __syncwarp();
        if (lane < kScanThreads / 32) warp_sums[lane] = wb;
        if (lane == kScanThreads / 32 - 1) warp_sums[kScanThreads / 32] = wi;
    }
    __syncthreads();
    const uint32_t r = add_to<SAT>(warp_sums[warp], before);
    *total = warp_sums[kScanThreads / 32];
    __syncthreads();
    return r;
}

// A radix sort's work: pairs on the device, their capacity, digits of a pass.
struct SortCount {
    const uint32_t *pairs;
    uint32_t cap, digits;
};
constexpr int kRadixThreads = 256;
constexpr int kRadixItems = 8;  // per thread
constexpr int kRadixTile = kRadixThreads * kRadixItems;
__host__ __device__ __forceinline__ uint32_t radix_blocks(uint32_t pairs)
{
    return pairs / kRadixTile + (pairs % kRadixTile ? 1u : 0u);
}

// Single-pass exclusive scan with decoupled look-back (Merrill and Garland, "Single-pass
// Parallel Prefix Scan with Decoupled Look-back", 2016). Blocks take their tile of kScanTile
// values in the order they start (a ticket), publish the tile's sum, then walk back over
// the tiles before theirs, 32 at a time, adding published sums until one publishes its
// inclusive prefix.
// A tile's status word: (flag << 32) | value, flag 0 = nothing yet, 1 = the tile's sum,
// 2 = the inclusive prefix through the tile; written whole, so a reader sees one or the other.
// A tile before a block's own was taken by a block that started earlier and publishes its sum
// without waiting, so every wait ends; each is still bounded (kScanWaitLimit reads) and a
// wait that runs out is recorded in the debug status word and counts the tile as empty.
constexpr uint32_t kScanWaitLimit = 1u << 24;
constexpr uint64_t kScanSum = 1ull << 32, kScanPrefix = 2ull << 32;

__device__ __forceinline__ uint64_t ld_status(const uint64_t *p) { return *(const volatile uint64_t *)p; }
__device__ __forceinline__ void st_status(uint64_t *p, uint64_t v) { *(volatile uint64_t *)p = v; }

// With `sort` the values are a digit histogram's, a column per tile of the pairs there are (n: of as
// many as fit), and the blocks past them leave at once.
template <bool SAT>
__global__ void __launch_bounds__(kScanThreads) k_scan(const uint32_t *in, uint32_t *out, uint32_t n,
                                                      uint64_t *status, uint32_t *ticket, uint32_t *total_dev,
                                                      uint32_t *debug, const uint32_t *rec_total, uint32_t *host,
                                                      SortCount sort)
{
    __shared__ uint32_t s_tile, s_prefix;
    if (threadIdx.x == 0) s_tile = gridDim.x == 1 ? 0u : atomicAdd(ticket, 1u);
    if (sort.pairs) n = radix_blocks(min(__ldg(sort.pairs), sort.cap)) * sort.digits;
    __syncthreads();
    const uint32_t tile = s_tile;
    if (sort.pairs && (uint64_t)tile * kScanTile >= n) return;
    const uint32_t base = tile * (uint32_t)kScanTile + threadIdx.x * kScanItems;
    // each thread's 8 values as two 16-byte words (base is a multiple of 8 words)
    uint32_t v[kScanItems];
    if (base + kScanItems <= n) {
        const uint4 a = *reinterpret_cast<const uint4 *>(in + base), b = *reinterpret_cast<const uint4 *>(in + base + 4);
        v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
    } else {
#pragma unroll
        for (int i = 0; i < kScanItems; i++) v[i] = (base + i < n) ? in[base + i] : 0u;
    }
    uint32_t sum = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; i++) sum = add_to<SAT>(sum, v[i]);
    uint32_t agg;
    uint32_t run = block_excl_scan<SAT>(sum, &agg);
    if (threadIdx.x < 32) {
        // warp 0 looks back 32 tiles at a time: lane k reads the status of tile (window - k)
        const uint32_t lane = threadIdx.x;
        uint32_t prefix = 0;
        if (tile == 0) {
            if (lane == 0) st_status(status, kScanPrefix | agg);
        } else {
            if (lane == 0) st_status(status + tile, kScanSum | agg);
            for (int64_t win = (int64_t)tile - 1;; win -= 32) {
                const int64_t p = win - (int64_t)lane;
                uint64_t st = p >= 0 ? ld_status(status + p) : kScanPrefix;  // before tile 0: a zero prefix
                for (uint32_t w = 0; !__all_sync(0xffffffffu, (st >> 32) != 0);) {
                    if (++w < kScanWaitLimit) {
                        if ((st >> 32) == 0) st = ld_status(status + p);
                    } else if ((st >> 32) == 0) {
                        st = kScanSum;  // counted as empty
                        if (debug) atomicCAS(debug, 0u, (uint32_t)DBG_SCAN_WAIT);
                    }
                }
                // the nearest tile with its inclusive prefix ends the walk; the nearer ones add sums
                const uint32_t prefixed = __ballot_sync(0xffffffffu, (st >> 32) == 2);
                const uint32_t upto = prefixed ? (uint32_t)__ffs(prefixed) - 1u : 31u;
                uint32_t add = lane <= upto ? (uint32_t)st : 0u;
                if (SAT) {  // in halves, whose 32 sums fit
                    const uint32_t lo = __reduce_add_sync(0xffffffffu, add & 0xFFFFu);
                    const uint32_t hi = __reduce_add_sync(0xffffffffu, add >> 16) + (lo >> 16);
                    add = hi > 0xFFFFu ? 0xFFFFFFFFu : (hi << 16) | (lo & 0xFFFFu);
                } else {
                    add = __reduce_add_sync(0xffffffffu, add);
                }
                prefix = add_to<SAT>(prefix, add);
                if (prefixed) break;
            }
            if (lane == 0) st_status(status + tile, kScanPrefix | add_to<SAT>(prefix, agg));
        }
        if (lane == 0) {
            s_prefix = prefix;
            if (tile + 1 == gridDim.x) {
                *total_dev = add_to<SAT>(prefix, agg);
                if (host) {  // page-locked: the pass's record and pair totals, without a copy behind it
                    host[0] = rec_total[0];
                    host[1] = rec_total[1];  // an ordered pass's is this scan's
                }
            }
        }
    }
    __syncthreads();
    run = add_to<SAT>(run, s_prefix);
    uint32_t o[kScanItems];
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        o[i] = run;
        run = add_to<SAT>(run, v[i]);
    }
    if (base + kScanItems <= n) {
        *reinterpret_cast<uint4 *>(out + base) = make_uint4(o[0], o[1], o[2], o[3]);
        *reinterpret_cast<uint4 *>(out + base + 4) = make_uint4(o[4], o[5], o[6], o[7]);
    } else {
#pragma unroll
        for (int i = 0; i < kScanItems; i++)
            if (base + i < n) out[base + i] = o[i];
    }
}

size_t scan_temp_words(uint32_t n)
{
    // a 64-bit status word per tile, then the ticket
    return 2 * (((size_t)n + kScanTile - 1) / kScanTile) + 64;
}

template <bool SAT>
static int start_scan(const uint32_t *in, uint32_t *out, uint32_t n, uint32_t *temp, uint32_t *total_dev, uint32_t *debug,
                      cudaStream_t s, const uint32_t *rec_total, uint32_t *host, SortCount sort, bool temp_zeroed = false)
{
    if (n == 0) {
        cudaMemsetAsync(total_dev, 0, sizeof(uint32_t), s);
        return 0;
    }
    const uint32_t nb = (n + kScanTile - 1) / kScanTile;
    // temp is 8-byte aligned (scratch slices start on 256-byte boundaries); a single tile needs
    // neither tickets nor statuses (and so no clearing)
    uint64_t *status = reinterpret_cast<uint64_t *>(temp);
    uint32_t *ticket = temp + 2 * (size_t)nb;
    if (nb > 1 && !temp_zeroed) cudaMemsetAsync(temp, 0, (2 * (size_t)nb + 1) * sizeof(uint32_t), s);
    k_scan<SAT><<<nb, kScanThreads, 0, s>>>(in, out, n, status, ticket, total_dev, debug, rec_total, host, sort);
    return 1;
}

int launch_scan(const uint32_t *in, uint32_t *out, uint32_t n, uint32_t *temp, uint32_t *total_dev, uint32_t *debug,
                cudaStream_t s, const uint32_t *rec_total, uint32_t *host)
{
    return start_scan<true>(in, out, n, temp, total_dev, debug, s, rec_total, host, SortCount{nullptr, 0u, 0u});
}

// ------------------------------------------------------------------ record -> tiles
//
// Three kernels run over the (record, tile of its box) candidates: the occlusion bounds, the
// pair count and the pair writes. Boxes hold from one tile to thousands, so a warp takes 32
// records, each lane sets one up into shared memory (BoxRec), and the warp then runs over the
// candidates of all 32 in order, 32 at a time, each lane finding its candidate's record in the
// prefix sums of the tile counts: every lane has a candidate whatever the boxes are. Passes of
// few records (full-screen quads, sprites) split a group's candidates over several warps in
// contiguous parts. Both keep submission order: a part's pairs follow the earlier parts'.

constexpr int kRecWarps = 4;  // warps per CTA of the record kernels

__device__ __forceinline__ uint32_t records_in(const BinArgs &A) { return min(*A.nrec_dev, A.nrec); }

// the frame that owns tile t: the last whose first tile is at or before it
__device__ __forceinline__ uint32_t frame_of_tile(const BinArgs &A, uint32_t t)
{
    uint32_t lo = 0, hi = A.nframes - 1;
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (A.frames[mid].tile_base <= t) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// A triangle record's edges as integers for an exact test over pixels [xl, xh] x [yl, yh]:
// edge k is (x - iax) * a - (y - iay) * b, sign-flipped for a negative area so that covered
// means >= 0. The record's positions and per-edge differences are integer-valued floats; when
// every product (px - ax) * A, (py - ay) * B that the per-pixel test (raster.c:299-302,
// 534-536) forms there is below 2^24 in magnitude, those products are exact, so each edge
// function's sign per pixel is the sign of the exact integer. False when one could be inexact.
__device__ __forceinline__ bool exact_edges(const float4 &q0, const float4 &q1, const float4 &q12, const float4 &q13,
                                            bool pos, int xl, int xh, int yl, int yh, int *iax, int *iay, int *a, int *b)
{
    const float ax[3] = {q0.z, q1.x, q0.x}, ay[3] = {q0.w, q1.y, q0.y};
    const float ea[3] = {q12.y, q12.w, q13.y}, eb[3] = {q12.z, q13.x, q13.z};
    bool ok = true;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        constexpr float kLim = 16777216.0f;  // 2^24
        ok = ok && fabsf(ax[k]) < kLim && fabsf(ay[k]) < kLim && fabsf(ea[k]) < kLim && fabsf(eb[k]) < kLim;
        iax[k] = (int)ax[k];
        iay[k] = (int)ay[k];
        a[k] = pos ? (int)ea[k] : -(int)ea[k];
        b[k] = pos ? (int)eb[k] : -(int)eb[k];
        const long long mx = max(llabs((long long)xl - iax[k]), llabs((long long)xh - iax[k])) * llabs((long long)a[k]);
        const long long my = max(llabs((long long)yl - iay[k]), llabs((long long)yh - iay[k])) * llabs((long long)b[k]);
        ok = ok && mx < (1ll << 24) && my < (1ll << 24);
    }
    return ok;
}

__device__ __forceinline__ bool has_depth_bound(uint32_t flags)
{
    const uint32_t zc = (flags >> 1) & 3u;
    return ((flags >> kRecTypeShift) & 3u) == REC_TRI && (zc == ZC_LESS || zc == ZC_LEQUAL);
}

// A record's candidate tiles, row-major: `w` per row from (tx0, ty0).
enum BoxMode : uint32_t {
    BOX_TEST = 1u,  // some tile may fail the edge test: e00 + col * sx - row * sy per edge decides
    BOX_HIDE = 2u,  // the tile's occlusion bound may hide the record
};
struct BoxRec {
    int tx0, ty0, w;
    uint32_t mode;
    int e00[3];
    float dmin;              // lower bound of the record's depths
    int sx[3];
    uint32_t mn;             // the record's box in pixels, x | y << 16
    int sy[3];
    uint32_t mx;
    float4 zp;               // depth plane
    uint32_t tile0, tiles_x; // global tile id at (tx0, ty0), tiles per row of its frame
    float inv_w;
    uint32_t pad;
};
static_assert(sizeof(BoxRec) % 16 == 0, "16-byte shared-memory words");

__device__ __forceinline__ uint32_t pack_xy(int x, int y) { return (uint32_t)x | ((uint32_t)y << 16); }

constexpr int kTestMinTiles = 4;  // smaller boxes keep every tile: little to drop, and the set-up dominates

// Sets up record r; returns its candidate count. OCCLUDE: the tiles it may cover whole.
// Otherwise the tiles of its box; the pairs are those where its coverage test can pass (a tile
// in which some edge function is negative at its largest, a corner, holds no covered pixel),
// less the hidden ones; points, lines and small boxes keep every tile not hidden.
template <bool OCCLUDE>
__device__ __forceinline__ int box_of(const BinArgs &A, uint32_t r, BoxRec &t)
{
    const float4 *q = reinterpret_cast<const float4 *>(A.records + (size_t)r * kRecWords);
    const float4 q1 = __ldg(q + 1), q2 = __ldg(q + 2), q12 = __ldg(q + 12), q13 = __ldg(q + 13);
    const DevFrame &F = A.frames[min(__float_as_uint(q13.w), A.nframes - 1)];
    const int sh = A.tile_shift, ts = 1 << sh;
    const int W = F.dims.width, H = F.dims.height;
    // set-up clamps every box to its framebuffer; the clamps here only keep tile indices inside
    // the frame's grid whatever a record holds
    const int mnx = min(max(__float_as_int(q1.z), 0), W - 1), mny = min(max(__float_as_int(q1.w), 0), H - 1);
    const int mxx = max(min(__float_as_int(q2.x), W - 1), mnx), mxy = max(min(__float_as_int(q2.y), H - 1), mny);
    const uint32_t flags = __float_as_uint(q12.x);
    const bool bounded = A.tile_near && F.occlude && has_depth_bound(flags);
    const float area = q2.z;
    int tx1, ty1;
    if (OCCLUDE) {
        // the tiles wholly inside the box, whose right and bottom sides may be the framebuffer's
        t.tx0 = (mnx + ts - 1) >> sh;
        t.ty0 = (mny + ts - 1) >> sh;
        tx1 = mxx == W - 1 ? (W - 1) >> sh : ((mxx + 1) >> sh) - 1;
        ty1 = mxy == H - 1 ? (H - 1) >> sh : ((mxy + 1) >> sh) - 1;
        if (!bounded || tx1 < t.tx0 || ty1 < t.ty0 || !(area > 0.0f || area < 0.0f)) return 0;
        t.zp = __ldg(q + 14);
        if (!isfinite(t.zp.w)) return 0;  // no plane
    } else {
        t.tx0 = mnx >> sh;
        t.ty0 = mny >> sh;
        tx1 = mxx >> sh;
        ty1 = mxy >> sh;
    }
    t.w = tx1 - t.tx0 + 1;
    const int cnt = t.w * (ty1 - t.ty0 + 1);
    t.tile0 = F.tile_base + (uint32_t)(t.ty0 * F.dims.tiles_x + t.tx0);
    t.tiles_x = (uint32_t)F.dims.tiles_x;
    t.inv_w = 1.0f / (float)t.w;
    t.mn = pack_xy(mnx, mny);
    t.mx = pack_xy(mxx, mxy);
    t.mode = 0u;
    if (!OCCLUDE) {
        if (bounded) {
            t.mode = BOX_HIDE;
            t.dmin = __ldg(reinterpret_cast<const float *>(q) + R_DMIN);
            t.zp = __ldg(q + 14);
        }
        if (cnt < kTestMinTiles || ((flags >> kRecTypeShift) & 3u) != REC_TRI) return cnt;
        if (!(area > 0.0f) && !(area < 0.0f)) return 0;  // zero or NaN area: the test never passes
    }
    const float4 q0 = __ldg(q + 0);
    int iax[3], iay[3], a[3], b[3];
    const int xl = t.tx0 << sh, yl = t.ty0 << sh;
    if (!exact_edges(q0, q1, q12, q13, area > 0.0f, xl, (tx1 << sh) + ts - 1, yl, (ty1 << sh) + ts - 1, iax, iay, a, b))
        return OCCLUDE ? 0 : cnt;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        // (x - ax) * a - (y - ay) * b is largest over a tile at its right edge when a >= 0 and its
        // top row when b >= 0; smallest at the opposite corner
        const bool right = (a[k] >= 0) != OCCLUDE, bottom = (b[k] >= 0) == OCCLUDE;
        t.e00[k] = (xl + (right ? ts - 1 : 0) - iax[k]) * a[k] - (yl + (bottom ? ts - 1 : 0) - iay[k]) * b[k];
        t.sx[k] = a[k] * ts;
        t.sy[k] = b[k] * ts;
    }
    t.mode |= BOX_TEST;
    return cnt;
}

// the box's i-th candidate as a column and row
__device__ __forceinline__ void box_tile(const BoxRec &t, int i, int &col, int &row)
{
    // (i + 1/2) / w lies at least 1/(2w) from an integer, and the float result is within
    // i / w * 2^-22 of it: exact below 2^20
    row = i < (1 << 20) ? (int)(((float)i + 0.5f) * t.inv_w) : i / t.w;
    col = i - row * t.w;
}

// the record gets a pair in this tile
__device__ __forceinline__ bool tile_gets_pair(const BinArgs &A, const BoxRec &t, int col, int row)
{
    if (t.mode & BOX_TEST) {
        bool ok = true;
#pragma unroll
        for (int k = 0; k < 3; k++) ok = ok && t.e00[k] + col * t.sx[k] - row * t.sy[k] >= 0;
        if (!ok) return false;
    }
    if (!(t.mode & BOX_HIDE)) return true;
    const uint32_t bound = __ldg(A.tile_near + t.tile0 + (uint32_t)row * t.tiles_x + (uint32_t)col);
    const int sh = A.tile_shift, x = (t.tx0 + col) << sh, y = (t.ty0 + row) << sh, ts = 1 << sh;
    const int mnx = (int)(t.mn & 0xFFFFu), mny = (int)(t.mn >> 16), mxx = (int)(t.mx & 0xFFFFu), mxy = (int)(t.mx >> 16);
    const float lo = fmaxf(t.dmin, depth_plane_bound(t.zp, mnx, mny, max(x, mnx), min(x + ts - 1, mxx), max(y, mny),
                                                     min(y + ts - 1, mxy)));
    return near_key(lo) >= bound;  // else strictly beyond it: no fragment of the record survives the tile
}

// Occlusion bounds (frames with DevFrame::occlude: every passing fragment replaces colour and
// depth, and only nearer or equal ones pass). A triangle that covers every pixel of a tile
// leaves no stored depth there beyond its own largest depth in the tile, whatever else is
// drawn before or after it; so a record whose smallest depth in the tile is beyond that
// changes nothing there, and its pair is dropped. Coverage is the exact edge test at the
// tile's corners (clipped to the framebuffer and inside the record's box), the depths are the
// plane's bounds. The bound of a tile is the nearest such depth (near_key, atomicMax).
__device__ __forceinline__ void take_bound(const BinArgs &A, const BoxRec &t, int col, int row)
{
    const int sh = A.tile_shift, ts = 1 << sh;
    const int xl = (t.tx0 + col) << sh, yl = (t.ty0 + row) << sh;
    const int W = (int)(t.mx & 0xFFFFu) + 1, H = (int)(t.mx >> 16) + 1;  // the box holds the tile's pixels
    const int cx = max(xl + ts - W, 0), cy = max(yl + ts - H, 0);        // those beyond the framebuffer
    bool all = true;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        // the corner moves in by the clipped pixels
        const int e = t.e00[k] + col * t.sx[k] - row * t.sy[k] + max(-(t.sx[k] >> sh), 0) * cx +
                      max(t.sy[k] >> sh, 0) * cy;
        all = all && e >= 0;
    }
    if (!all) return;
    const float up = depth_plane_upper(t.zp, (int)(t.mn & 0xFFFFu), (int)(t.mn >> 16), xl, xl + ts - 1 - cx, yl,
                                       yl + ts - 1 - cy);
    if (!(up < INFINITY)) return;
    const uint32_t key = near_key(up);
    uint32_t *at = A.tile_near + t.tile0 + (uint32_t)row * t.tiles_x + (uint32_t)col;
    // most records of a deep tile are not the nearest by then: look before the atomic (an old
    // value only costs an atomic)
    if (key > __ldcg(at)) atomicMax(at, key);
}

// The passes over the candidates: occlusion bounds; pairs per unit and the pair writes (ordered
// passes, sorted by tile afterwards); and, for order-free passes (k_tile_free.cu), the pairs in
// one go, in whatever order they come: each takes its rank in its tile's list as it is
// counted, and k_bin_place moves it there once the tiles' starts are scanned.
enum RecPass { PASS_OCCLUDE, PASS_COUNT, PASS_EXPAND, PASS_PAIRS };

// PASS_PAIRS: kept pairs collect in shared memory and leave 64 at a time, so that the one
// counter all warps share and the wait for a rank are paid per 64 pairs, by full warps (of a
// deep frame's candidates one in fifty is kept).
constexpr uint32_t kQueueFlush = 64, kQueue = kQueueFlush + 32;

__device__ __forceinline__ void flush_pairs(const BinArgs &A, const uint2 *queue, uint32_t n)
{
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t pos = 0;
    if (lane == 0) pos = atomicAdd(A.total_dev, n);
    uint2 q[kQueueFlush / 32];
    uint32_t rank[kQueueFlush / 32];
#pragma unroll
    for (uint32_t k = 0; k < kQueueFlush / 32; k++)
        if (k * 32 + lane < n) {
            q[k] = queue[k * 32 + lane];
            rank[k] = atomicAdd(A.tile_count + q[k].x, 1u);
        }
    // Past the capacity the exact total serves nothing, and would wrap: an addition that finds it
    // exceeded is taken back, so that it stays exceeded and below the capacity (at most kMaxEntries)
    // and 64 for every resident warp, far from 2^32. (Looked at here, with the ranks on their way.)
    if (lane == 0 && pos > A.npairs) atomicSub(A.total_dev, n);
    pos = __shfl_sync(0xffffffffu, pos, 0) + lane;
#pragma unroll
    for (uint32_t k = 0; k < kQueueFlush / 32; k++, pos += 32)
        if (k * 32 + lane < n && pos < A.npairs) {
            A.keys[pos] = q[k].x;
            A.vals_alt[pos] = q[k].y;
            A.keys_alt[pos] = rank[k];
        }
}

template <RecPass PASS>
__global__ void __launch_bounds__(kRecWarps * 32) k_bin_records(BinArgs A)
{
    __shared__ BoxRec s_box[kRecWarps][32];
    __shared__ uint32_t s_end[kRecWarps][32];  // inclusive sums of the candidate counts
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, below = (1u << lane) - 1u;
    const uint32_t n = records_in(A);
    __shared__ uint2 s_queue[PASS == PASS_PAIRS ? kRecWarps : 1][PASS == PASS_PAIRS ? kQueue : 1];  // tile, record
    uint32_t queued = 0;
    const BoxRec *box = s_box[warp];
    const uint32_t *ends = s_end[warp];
    if (PASS == PASS_PAIRS && A.tile_frame)
        for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < A.ntiles; t += gridDim.x * blockDim.x)
            A.tile_frame[t] = frame_of_tile(A, t);
    // the host's units are for the record capacity: fewer records take more warps each
    uint32_t wpg = 1;
    while (wpg < 32u && ((n + 31u) / 32u) * wpg * 2u <= A.units) wpg *= 2;
    for (uint32_t u = blockIdx.x * kRecWarps + warp; u < A.units; u += gridDim.x * kRecWarps) {
        // unit u: part u % wpg of the candidates of records [r0, r0 + 32)
        const uint32_t r0 = u / wpg * 32u, part = u % wpg;
        uint32_t kept = 0;
        if (r0 < n) {
            BoxRec b;
            const int cnt = r0 + lane < n ? box_of<PASS == PASS_OCCLUDE>(A, r0 + lane, b) : 0;
            const uint32_t incl = warp_incl_scan((uint32_t)cnt);
            const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
            if (cnt) s_box[warp][lane] = b;
            s_end[warp][lane] = incl;
            __syncwarp();
            const uint32_t per = ((total + wpg - 1) / wpg + 31u) & ~31u;
            const uint32_t lo = min(part * per, total), hi = min(lo + per, total);
            const uint32_t at = PASS == PASS_EXPAND ? A.rec_tiles[u] : 0u;
            // the lane's current record and its candidates [first, end): a box of many tiles
            // serves many steps before the next search
            uint32_t j = 0, first = 0, end = 0;
            for (uint32_t c0 = lo; c0 < hi; c0 += 32) {
                const uint32_t c = c0 + lane;
                bool get = false;
                uint32_t tile = 0;
                if (c < hi) {
                    if (c >= end) {  // the record: the first whose inclusive sum exceeds c
                        j = 0;
#pragma unroll
                        for (uint32_t step = 16; step; step >>= 1)
                            if (ends[j + step - 1] <= c) j += step;
                        first = j ? ends[j - 1] : 0u;
                        end = ends[j];
                    }
                    const BoxRec &t = box[j];
                    int col, row;
                    box_tile(t, (int)(c - first), col, row);
                    if (PASS == PASS_OCCLUDE) {
                        take_bound(A, t, col, row);
                    } else {
                        get = tile_gets_pair(A, t, col, row);
                        tile = t.tile0 + (uint32_t)row * t.tiles_x + (uint32_t)col;
                        get = debug_check(A.debug, tile < A.ntiles, DBG_BIN_TILE) && get;
                    }
                }
                if (PASS == PASS_OCCLUDE) continue;
                const uint32_t m = __ballot_sync(0xffffffffu, get);
                if (PASS == PASS_EXPAND && get) {
                    const uint32_t pos = at + kept + (uint32_t)__popc(m & below);
                    if (pos < A.npairs) {
                        A.keys[pos] = tile;
                        A.vals[pos] = r0 + j;
                    }
                }
                if (PASS == PASS_PAIRS && m) {
                    if (get) s_queue[warp][queued + (uint32_t)__popc(m & below)] = make_uint2(tile, r0 + j);
                    queued += (uint32_t)__popc(m);
                    __syncwarp();
                    if (queued >= kQueueFlush) {
                        flush_pairs(A, s_queue[warp], kQueueFlush);
                        queued -= kQueueFlush;
                        const uint2 rest = s_queue[warp][kQueueFlush + lane];  // fewer than 32
                        __syncwarp();
                        if (lane < queued) s_queue[warp][lane] = rest;
                        __syncwarp();
                    }
                }
                kept += (uint32_t)__popc(m);
            }
            __syncwarp();
        }
        if (PASS == PASS_COUNT && lane == 0) A.rec_tiles[u] = kept;  // units past the records: none
    }
    if (PASS == PASS_PAIRS && queued) flush_pairs(A, s_queue[warp], queued);
}

// Order-free passes: each pair's record to its place in its tile's list.
__global__ void __launch_bounds__(256) k_bin_place(BinArgs A)
{
    const uint32_t n = *A.total_dev;
    if (n > A.npairs) return;  // the tile launch leaves the frames alone then
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t at = __ldg(A.tile_start + A.keys[i]) + A.keys_alt[i];
        if (at < A.npairs) A.vals[at] = A.vals_alt[i];
    }
}

// grids cover the work or the GPU (16 CTAs per SM), whichever is smaller; kernels loop over the rest
unsigned stride_grid(uint64_t threads, unsigned block, int sms)
{
    const uint64_t want = (threads + block - 1) / block;
    const uint64_t cap = (uint64_t)(sms > 0 ? sms : 1) * 16;
    return (unsigned)std::max<uint64_t>(1, std::min(want, cap));
}

// Where the sorted tile id changes, the earlier tile's range ends and the later one's
// starts: the first writes the end position into tile_count, the second its start.
__global__ void __launch_bounds__(256) k_tile_bounds(BinArgs A)
{
    const uint32_t n = min(*A.total_dev, A.npairs);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t k = A.keys[i];
        if (!debug_check(A.debug, k < A.ntiles, DBG_BIN_TILE)) continue;
        if (i == 0 || A.keys[i - 1] != k) A.tile_start[k] = i;
        if (i + 1 == n || A.keys[i + 1] != k) A.tile_count[k] = i + 1;
    }
}

// end position - start = count; a tile without pairs has both still zero. Also the frame
// that owns each tile, so the tile kernel reads it instead of searching the frame table per
// tile.
__global__ void __launch_bounds__(256) k_tile_counts(BinArgs A)
{
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < A.ntiles; t += gridDim.x * blockDim.x) {
        A.tile_count[t] -= A.tile_start[t];
        if (A.tile_frame) A.tile_frame[t] = frame_of_tile(A, t);
    }
}

int launch_tile_ranges(const BinArgs &a, cudaStream_t s)
{
    if (a.npairs) k_tile_bounds<<<stride_grid(a.npairs, 256, a.sms), 256, 0, s>>>(a);
    k_tile_counts<<<stride_grid(a.ntiles, 256, a.sms), 256, 0, s>>>(a);
    return a.npairs ? 2 : 1;
}

// Work units for up to nrec records: the groups of 32 alone fill the GPU (64 warps per SM) from
// about 300,000 records up; fewer groups split their candidates, up to 32 ways.
uint32_t bin_units(uint32_t nrec, int sms)
{
    const uint32_t groups = (nrec + 31u) / 32u, warps = (uint32_t)(sms > 0 ? sms : 1) * 64u;
    uint32_t k = 1;
    while (k < 32 && (uint64_t)groups * k < warps) k *= 2;
    return groups * k;
}

namespace {

template <RecPass PASS>
int launch_records(const BinArgs &a, cudaStream_t s)
{
    k_bin_records<PASS><<<stride_grid((uint64_t)a.units * 32, kRecWarps * 32, 2 * a.sms), kRecWarps * 32, 0, s>>>(a);
    return 1;
}

}  // namespace

int launch_bin_count(const BinArgs &a, cudaStream_t s)
{
    if (!a.nrec) return 0;
    const int occlude = a.tile_near ? launch_records<PASS_OCCLUDE>(a, s) : 0;
    if (!a.order_free) return occlude + launch_records<PASS_COUNT>(a, s) +
                              launch_scan(a.rec_tiles, a.rec_tiles, a.units, a.scan_temp, a.total_dev, a.debug, s, a.nrec_dev,
                                          a.totals_host);
    return occlude + launch_records<PASS_PAIRS>(a, s) +
           start_scan<false>(a.tile_count, a.tile_start, a.ntiles, a.scan_temp, a.sort_total_dev, a.debug, s, a.nrec_dev,
                             a.totals_host, SortCount{nullptr, 0u, 0u}, true);
}

int launch_bin_expand(const BinArgs &a, cudaStream_t s)
{
    if (!a.nrec) return 0;
    if (!a.order_free) return launch_records<PASS_EXPAND>(a, s);
    k_bin_place<<<stride_grid(std::min<uint32_t>(a.npairs, 1u << 20), 256, a.sms), 256, 0, s>>>(a);
    return 1;
}

// ------------------------------------------------------------------ work order of the tile launch

// coarse log2 bucket of a tile's record count: 8 steps per octave, 0 for an empty tile
__device__ __forceinline__ uint32_t cost_bucket(uint32_t c)
{
    if (c == 0) return 0;
    const int lg = 31 - __clz(c);
    const uint32_t frac = lg >= 3 ? (c >> (lg - 3)) & 7u : (c << (3 - lg)) & 7u;
    return min(1u + (uint32_t)lg * 8u + frac, 255u);
}

// aux[0..255]: tiles per bucket; aux[256..511]: placement cursors; all zero at launch
__global__ void __launch_bounds__(256) k_order_hist(const uint32_t *tile_count, uint32_t ntiles, uint32_t *aux)
{
    __shared__ uint32_t h[256];
    h[threadIdx.x] = 0;
    __syncthreads();
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < ntiles; t += gridDim.x * blockDim.x)
        atomicAdd(&h[cost_bucket(tile_count[t])], 1u);
    __syncthreads();
    if (h[threadIdx.x]) atomicAdd(&aux[threadIdx.x], h[threadIdx.x]);
}

// Places every tile after all tiles of costlier buckets. The order inside a bucket is whatever
// the atomics give: tiles are independent, so it changes timing only.
__global__ void __launch_bounds__(256) k_order_scatter(const uint32_t *tile_count, uint32_t ntiles, uint32_t *aux,
                                                       uint32_t *order)
{
    __shared__ uint32_t start[256];
    __shared__ uint32_t warp_tot[8];
    const int e = 255 - (int)threadIdx.x;  // costliest first
    const uint32_t v = aux[e];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t x = warp_incl_scan(v);
    if (lane == 31) warp_tot[warp] = x;
    __syncthreads();
    uint32_t before = 0;
    for (int w = 0; w < warp; w++) before += warp_tot[w];
    start[e] = before + x - v;
    __syncthreads();
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < ntiles; t += gridDim.x * blockDim.x) {
        const uint32_t k = cost_bucket(tile_count[t]);
        order[start[k] + atomicAdd(&aux[256 + k], 1u)] = t;
    }
}

int launch_tile_order(const uint32_t *tile_count, uint32_t ntiles, uint32_t *aux, uint32_t *order, int sms,
                      cudaStream_t s)
{
    if (!ntiles) return 0;
    cudaMemsetAsync(aux, 0, kOrderAuxWords * sizeof(uint32_t), s);
    const unsigned g = stride_grid(ntiles, 256, sms);
    k_order_hist<<<g, 256, 0, s>>>(tile_count, ntiles, aux);
    k_order_scatter<<<g, 256, 0, s>>>(tile_count, ntiles, aux, order);
    return 2;
}

// ------------------------------------------------------------------ stable radix sort by tile

// The grids and the scratch are for the capacity, the work for the pairs there are: blocks step
// through the tiles of kRadixTile pairs, and a pass's histogram has a column per tile in use. (A
// context's capacity is its largest pass's: 40 blended quads after a pass of two million in the
// same context, whole passes: 371 us with a histogram of the capacity, 267 so, 255 in a context
// of their own.)
constexpr int kRadixWarps = kRadixThreads / 32;
constexpr int kRadixDigits = 512;  // up to 9-bit digits; a sort uses ceil(bits / 9) balanced passes

size_t radix_hist_words(uint32_t npairs)
{
    return (size_t)radix_blocks(npairs) * kRadixDigits + 64;
}

__global__ void __launch_bounds__(kRadixThreads) k_radix_hist(const uint32_t *keys, uint32_t cap,
                                                             const uint32_t *n_dev, int shift, uint32_t mask,
                                                             uint32_t *hist)
{
    const uint32_t n = min(*n_dev, cap), nblocks = radix_blocks(n);
    const int ndig = (int)mask + 1;
    __shared__ uint32_t h[kRadixDigits];
    for (uint32_t b = blockIdx.x; b < nblocks; b += gridDim.x) {
        for (int i = threadIdx.x; i < ndig; i += kRadixThreads) h[i] = 0;
        __syncthreads();
        const uint32_t base = b * (uint32_t)kRadixTile;
#pragma unroll
        for (int k = 0; k < kRadixItems; k++) {
            const uint32_t i = base + k * kRadixThreads + threadIdx.x;
            if (i < n) atomicAdd(&h[(keys[i] >> shift) & mask], 1u);
        }
        __syncthreads();
        for (int d = threadIdx.x; d < ndig; d += kRadixThreads) hist[(size_t)d * nblocks + b] = h[d];
    }
}

// Stable scatter: warp w owns items [w*256, w*256+256) of the block, taken 32 at a time in
// order; match-any groups equal digits, the leader advances the warp's digit counter, and
// per-digit prefix sums over warps and blocks place every item after all earlier ones. The
// block first sorts its items by digit in shared memory, so that each digit's run leaves
// as consecutive addresses (coalesced writes) rather than one scattered word per item.
__global__ void __launch_bounds__(kRadixThreads) k_radix_scatter(const uint32_t *keys, const uint32_t *vals,
                                                                uint32_t cap, const uint32_t *n_dev, int shift,
                                                                uint32_t mask,
                                                                const uint32_t *hist_scan,
                                                                uint32_t *keys_out, uint32_t *vals_out)
{
    __shared__ uint32_t wcount[kRadixWarps][kRadixDigits];  // per warp and digit: count, then block-local start
    __shared__ uint32_t dstart[kRadixDigits];                // block-local start of each digit's run
    __shared__ uint32_t gdelta[kRadixDigits];                // global start minus block-local start
    __shared__ uint32_t skey[kRadixTile], sval[kRadixTile];
    __shared__ uint32_t wsum[kRadixWarps];
    const uint32_t n = min(*n_dev, cap), nblocks = radix_blocks(n);
    const int ndig = (int)mask + 1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    for (uint32_t b = blockIdx.x; b < nblocks; b += gridDim.x) {
        if (b != blockIdx.x) __syncthreads();  // the previous tile's pairs have left
        for (int i = threadIdx.x; i < kRadixWarps * kRadixDigits; i += kRadixThreads) (&wcount[0][0])[i] = 0;
        __syncthreads();
        const uint32_t bbase = b * (uint32_t)kRadixTile;
        const uint32_t wbase = bbase + warp * 32 * kRadixItems;
        uint32_t key[kRadixItems], val[kRadixItems], rank[kRadixItems];
#pragma unroll
        for (int k = 0; k < kRadixItems; k++) {
            const uint32_t i = wbase + k * 32 + lane;
            const bool valid = i < n;
            key[k] = valid ? keys[i] : 0u;
            val[k] = valid ? vals[i] : 0u;
            const uint32_t d = valid ? ((key[k] >> shift) & mask) : 0xFFFFFFFFu;
            const uint32_t peers = __match_any_sync(0xffffffffu, d);
            const int leader = __ffs(peers) - 1;
            const uint32_t pre = valid ? wcount[warp][d] : 0u;
            __syncwarp();
            if (valid && lane == leader) wcount[warp][d] = pre + __popc(peers);
            __syncwarp();
            rank[k] = pre + __popc(peers & lt);
        }
        __syncthreads();
        // per digit: the block's count, then each warp's start within the digit's run
        for (int d = threadIdx.x; d < kRadixDigits; d += kRadixThreads) {
            uint32_t run = 0;
#pragma unroll
            for (int w = 0; w < kRadixWarps; w++) {
                const uint32_t c = d < ndig ? wcount[w][d] : 0u;
                wcount[w][d] = run;
                run += c;
            }
            dstart[d] = run;  // the count for now
        }
        __syncthreads();
        // exclusive scan of the digit counts (512 entries, 2 per thread) into block-local starts
        {
            const int d0 = 2 * threadIdx.x;
            const uint32_t c0 = dstart[d0], c1 = dstart[d0 + 1];
            uint32_t incl = c0 + c1, x = incl;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            if (lane == 31) wsum[warp] = x;
            __syncthreads();
            uint32_t before = 0;
            for (int w = 0; w < warp; w++) before += wsum[w];
            const uint32_t excl = before + x - incl;
            __syncthreads();
            dstart[d0] = excl;
            dstart[d0 + 1] = excl + c0;
            if (d0 < ndig) gdelta[d0] = hist_scan[(size_t)d0 * nblocks + b] - excl;
            if (d0 + 1 < ndig) gdelta[d0 + 1] = hist_scan[(size_t)(d0 + 1) * nblocks + b] - (excl + c0);
        }
        __syncthreads();
        // items into shared memory in digit order (stable: warp order, then item order)
#pragma unroll
        for (int k = 0; k < kRadixItems; k++) {
            const uint32_t i = wbase + k * 32 + lane;
            if (i < n) {
                const uint32_t d = (key[k] >> shift) & mask;
                const uint32_t at = dstart[d] + wcount[warp][d] + rank[k];
                skey[at] = key[k];
                sval[at] = val[k];
            }
        }
        __syncthreads();
        // consecutive slots of one digit go to consecutive global positions
        const uint32_t valid_n = n > bbase ? min((uint32_t)kRadixTile, n - bbase) : 0u;
#pragma unroll
        for (int k = 0; k < kRadixItems; k++) {
            const uint32_t at = k * kRadixThreads + threadIdx.x;
            if (at < valid_n) {
                const uint32_t kk = skey[at];
                const uint32_t pos = gdelta[(kk >> shift) & mask] + at;
                keys_out[pos] = kk;
                vals_out[pos] = sval[at];
            }
        }
    }
}

int launch_bin_sort(BinArgs &a, cudaStream_t s)
{
    const uint32_t n = a.npairs;  // capacity; the kernels read the real count from total_dev
    if (n == 0) return 0;
    int launches = 0;
    int bits = 1;
    while (bits < 32 && (1u << bits) < a.ntiles) bits++;
    const int passes = (bits + 8) / 9;
    const int width = (bits + passes - 1) / passes;  // balanced digits of at most 9 bits
    const uint32_t nb = radix_blocks(n), grid = std::min<uint32_t>(nb, 16u * (uint32_t)std::max(1, a.sms));
    for (int shift = 0; shift < bits; shift += width) {
        const int nbits = (bits - shift) < width ? (bits - shift) : width;
        const uint32_t mask = (1u << nbits) - 1u;
        k_radix_hist<<<grid, kRadixThreads, 0, s>>>(a.keys, n, a.total_dev, shift, mask, a.radix_hist);
        launches += 2 + start_scan<false>(a.radix_hist, a.radix_hist, nb * (mask + 1u), a.scan_temp, a.sort_total_dev, a.debug, s,
                                          nullptr, nullptr, SortCount{a.total_dev, n, mask + 1u});
        k_radix_scatter<<<grid, kRadixThreads, 0, s>>>(a.keys, a.vals, n, a.total_dev, shift, mask, a.radix_hist,
                                                       a.keys_alt, a.vals_alt);
        uint32_t *tk = a.keys, *tv = a.vals;
        a.keys = a.keys_alt;
        a.vals = a.vals_alt;
        a.keys_alt = tk;
        a.vals_alt = tv;
    }
    return launches;
}

}  // namespace mtgl
