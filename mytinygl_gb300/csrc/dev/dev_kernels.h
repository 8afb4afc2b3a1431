// dev_kernels.h — host-side launchers of the sm_103a kernels (one translation unit each).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "mtgl_device.cuh"

namespace mtgl {

constexpr uint32_t kClipClasses = 96;  // one-plane candidates: first plane x in/out pattern; the rest
// Each class is counted in kClipSlots counters (a block of the count pass uses slot
// blockIdx % kClipSlots), so that the appends of many blocks do not all meet on a few words.
constexpr uint32_t kClipSlots = 32;
constexpr int kDebugStatusWord = 8;  // word of an Exec's counters that the debug bounds checks write
constexpr uint32_t kClipBuckets = kClipClasses * kClipSlots;  // class-major

struct GeomArgs {
    const DevDraw *draws;
    const uint32_t *draw_vslot_base;  // per draw, ascending
    const uint32_t *draw_tri_base;    // per draw, ascending
    int32_t ndraws;
    const mtgl_vertex_state *vstates;
    const DevRaster *rasters;
    PostVertices verts;
    PostEye *eyes;                    // null when no draw of the pass lights per fragment
    uint32_t total_slots;
    uint32_t total_tris;
    const DevFrame *frames;           // the raster state's `frame` indexes this table
    uint32_t nframes;
    uint32_t *tri_counts;             // count pass output
    const uint32_t *tri_offsets;      // emit pass input (exclusive scan of tri_counts)
    float *records;                   // emit pass output, kRecWords per record
    float *eye_records;               // emit pass output, kEyeWords per record (may be null)
    uint32_t records_cap;             // records the output buffers hold (writes beyond are dropped)
    uint32_t *clip_list;              // triangles that straddle a clip plane (total_tris entries)
    uint32_t *clip_class;             // per entry: bucket << 20 | rank within the bucket
    uint32_t *clip_sorted;            // the entries grouped by class (null: process clip_list as is)
    uint32_t *class_count;            // kClipBuckets counters (zeroed by the count launch)
    uint32_t *emit_list;              // primitives the set-up emit pass writes (count pass output; unordered)
    uint32_t *list_counts;            // entries of [0] the clip list, [1] the emit list (device; zeroed
                                      // by the count launch)
    int32_t sms;
    uint32_t *debug;                  // status word of the debug bounds checks
    // order-free set-up
    uint32_t *rec_total;              // records made, then the word of the pair total (device; both
                                      // zeroed by the vertex launch)
    uint32_t *rec_seq;                // per record: its place in the submission order
    uint32_t *zero;                   // words the vertex launch clears, beside list_counts and rec_total
    uint32_t zero_words;              // (0: none of them)
};

// K1: per-vertex stage (gl_api.c:263-348) for every vertex slot of the pass.
int launch_vertex(const GeomArgs &a, cudaStream_t s);
// K2: primitive assembly, clipping, perspective divide, culling and triangle setup
// (raster.c:451-529, 729-1017, 1199-1231); count pass then emit pass.
int launch_setup_count(const GeomArgs &a, cudaStream_t s);
int launch_setup_emit(const GeomArgs &a, cudaStream_t s);
// K2 of an order-free pass with record capacity: one pass, records in any order with their place
// in rec_seq. Without clip_sorted straddling triangles are clipped in the same launch.
int launch_setup_free(const GeomArgs &a, cudaStream_t s);
constexpr uint32_t kInlineClipTris = 16384;  // passes up to this many triangles do so

// Every launcher returns the number of kernels it launched.

// Device-wide exclusive scan of n uint32 values (in place allowed; one launch); writes the
// total to *total_dev. in and out 16-byte aligned; temp must hold scan_temp_words(n) words,
// 8-byte aligned; debug is the
// status word its bounded waits report to (may be null).
size_t scan_temp_words(uint32_t n);
// Sums stay at 2^32 - 1 instead of wrapping. With `host` (two page-locked words) the launch also
// writes rec_total[0] and [1], the pass's record and pair totals, there.
int launch_scan(const uint32_t *in, uint32_t *out, uint32_t n, uint32_t *temp, uint32_t *total_dev, uint32_t *debug,
                cudaStream_t s, const uint32_t *rec_total = nullptr, uint32_t *host = nullptr);

// The most records or pairs a pass may make: a larger total is refused (MTGL_ERR_OVERFLOW). Below
// 2^32 by more than the kernels' strides, so that their 32-bit loops end.
constexpr uint32_t kMaxEntries = 0xF0000000u;

// Element counts of the binning stage live on the device (written by the scans), so the
// stage runs without the host knowing them. `nrec` / `npairs` on the host are capacities:
// they size grids and buffers, and kernels read the real counts through nrec_dev / total_dev.
struct BinArgs {
    const float *records;
    uint32_t nrec;              // record capacity
    const uint32_t *nrec_dev;   // records written (may exceed nrec: the excess was dropped)
    const DevFrame *frames;
    uint32_t nframes;
    int32_t tile_shift;         // tile edge = 1 << tile_shift
    uint32_t ntiles;            // tiles of all frames
    uint32_t units;             // bin_units(nrec): work units of the record kernels
    uint32_t *rec_tiles;        // per unit its pair count, then the exclusive scan (in place)
    uint32_t *keys, *vals;      // pair buffers (capacity >= pairs)
    uint32_t *keys_alt, *vals_alt;
    uint32_t *tile_count;       // per tile (ntiles + 1 entries)
    uint32_t *tile_near;        // per tile: the occlusion bound (near_key; zero at launch); null when no
                                // frame of the pass has one
    uint32_t *tile_start;       // exclusive scan of tile_count
    uint32_t *tile_frame;       // per tile: the frame owning it, written with the tiles' ranges (null: one frame)
    uint32_t *radix_hist;       // radix histograms
    uint32_t *scan_temp;        // (zero at launch in order-free passes)
    uint32_t *total_dev;        // where the pair scan writes its total: the pairs generated
    uint32_t *totals_host;      // page-locked words that get the record and pair totals (may be null)
    uint32_t *sort_total_dev;   // a word the sort's histogram scans may overwrite
    int32_t order_free;         // tile lists need no order (k_tile_free.cu)
    uint32_t npairs;            // pair capacity of keys/vals (writes beyond are dropped)
    int32_t sms;                // SMs of the device (grid sizes)
    uint32_t *debug;            // status word of the debug bounds checks
};

// The count launch also takes the occlusion bounds first (where tile_near is given).
// Ordered passes: pairs per unit, scanned, and the pair total. Order-free passes: the pairs (tile
// in keys, record in vals_alt, rank in keys_alt), pairs per tile in tile_count and their scan in
// tile_start, and the total (*total_dev zero at launch); the expand launch then writes the lists.
int launch_bin_count(const BinArgs &a, cudaStream_t s);
uint32_t bin_units(uint32_t nrec, int sms);  // at most nrec + 31
int launch_bin_expand(const BinArgs &a, cudaStream_t s);
// Stable sort of (tile, record) pairs by tile; result in keys/vals. Uses keys_alt/vals_alt
// as ping-pong storage.
int launch_bin_sort(BinArgs &a, cudaStream_t s);
size_t radix_hist_words(uint32_t npairs);
// Each tile's range of the sorted pairs: tile_start and tile_count (zero for a tile with no
// pairs), read off the sorted keys where the tile id changes. tile_start and tile_count must
// be zero for every tile on entry.
int launch_tile_ranges(const BinArgs &a, cudaStream_t s);

// Work order of a tile launch, by descending record count (coarse log buckets), so that the
// longest tiles start first. order holds ntiles words, aux kOrderAuxWords.
int launch_tile_order(const uint32_t *tile_count, uint32_t ntiles, uint32_t *aux, uint32_t *order, int sms,
                      cudaStream_t s);
constexpr size_t kOrderAuxWords = 512;

struct TileArgs {
    const float *records;
    const float *eye_records;
    const uint32_t *rec_seq;     // order-free passes: a record's place in the submission order (null: its index)
    const uint32_t *tile_vals;   // record indices sorted by tile, submission order within a tile
    const uint32_t *tile_start;  // per tile
    const uint32_t *tile_count;
    const uint32_t *tile_frame;  // per tile: its frame (null: the pass has one)
    const DevRaster *rasters;
    uint32_t nrasters;
    const ClearOp *clears;       // all frames' clears; a frame holds its range
    const DevFrame *frames;
    uint32_t nframes;
    uint32_t ntiles;             // work items: global tile ids
    const uint32_t *order;       // item -> tile (null: item i is tile i)
    int32_t ctas;                // CTAs that step through the tiles (0: one per tile)
    int32_t tile_shift;
    int32_t any_texture;         // some raster state of the pass samples a texture
    int32_t any_stencil;         // some raster state of the pass tests the stencil
    // capacity check: when guard[0] > records_cap or guard[1] > pairs_cap the binning
    // dropped entries, and the launch leaves every framebuffer untouched
    const uint32_t *guard;
    uint32_t records_cap, pairs_cap;
    unsigned long long *fragments;
    int32_t defer;               // every record is a filled triangle with deferrable colour (k_tile.cuh)
    uint32_t *debug;             // status word of the debug bounds checks
    uint32_t entries_cap;        // entries tile_vals holds (debug bounds checks)
    int32_t order_free;          // the pass renders order-free (k_tile_free.cu)
};

// K4: per tile the clears, then its triangles through the full fragment pipeline
// (raster.c:532-724), then one write-back.
int launch_tile(const TileArgs &a, cudaStream_t s);
// resident CTAs per SM of the K4 variant a launch with these arguments uses
int tile_occupancy(const TileArgs &a);

// glClear without draws (gl_api.c:409-457)
void launch_clear(const ClearOp *ops_host, int nops, FrameDims dims, uint32_t *color, float *depth, uint8_t *stencil,
                  cudaStream_t s);
// packed RGBA8 texels from 1 (luminance), 2 (luminance, alpha) or 3 (RGB) bytes per texel
// (texture_upload_*, textures.c:141-269)
void launch_expand_texels(const uint8_t *raw, int comps, int64_t n, uint32_t *texels, cudaStream_t s);
// mip level 1 (textures.c:311-354)
void launch_mip1(const uint32_t *base, int32_t w, int32_t h, uint32_t *mip, cudaStream_t s);
// glDrawPixels blit (gl_api.c:1287-1376)
void launch_draw_pixels(const uint32_t *img, int32_t rx, int32_t ry, int32_t w, int32_t h, const DevRaster *raster,
                        FrameDims dims, uint32_t *color, float *depth, cudaStream_t s);

// Colour read-back by kernel into page-locked host memory mapped into the device's address
// space (dst is the device-side address): one launch per kReadbackMax items, the items in the
// launch's parameters. Returns the kernels launched.
struct ReadbackItem {
    const uint32_t *src;  // device colour buffer
    uint32_t *dst;        // device address of the host buffer
    uint32_t n;           // pixels
    uint32_t first_unit;  // set by the launcher
};
constexpr int kReadbackMax = 128;
constexpr uint32_t kReadbackUnit = 4096;  // pixels per work unit
struct ReadbackArgs {
    ReadbackItem item[kReadbackMax];
    int32_t count;
    uint32_t units;
};
int launch_readback(const ReadbackItem *items, int n, int sms, cudaStream_t s);

}  // namespace mtgl
