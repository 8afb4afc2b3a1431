// kernels.cu — stand-ins for the kernel launches: no pixel is computed. Each names itself in a log,
// the counting ones give the totals a test asks for, and the tile launch notes whether its guard
// let it write, and whether it writes the frame to the host too.
#include <string>

#include "dev_internal.h"

using namespace mtgl;

namespace {
uint32_t g_records, g_pairs;
std::string g_log;
int say(const char *what)
{
    if (!g_log.empty()) g_log += ' ';
    g_log += what;
    return 1;
}
}  // namespace

extern "C" {
void fake_totals(uint32_t records, uint32_t pairs)
{
    g_records = records;
    g_pairs = pairs;
}
const char *fake_log() { return g_log.c_str(); }
void fake_log_clear() { g_log.clear(); }
// whether binning may drop hidden pairs of a w x h frame of one opaque depth-tested triangle
int fake_occludes(int32_t w, int32_t h)
{
    mtgl_dev *d = nullptr;
    if (mtgl_dev_create(w, h, &d) != MTGL_OK) return -1;
    DevRaster R;
    memset(&R, 0, sizeof(R));
    R.rs.polygon_mode_front = R.rs.polygon_mode_back = GL_FILL;
    R.rs.depth_func = GL_LESS;
    R.depth_rejection = 1;
    R.fs.ctl = FC_DEPTH | FC_DEPTH_WRITE | FC_MASK_ALL;
    PendingDraw p;
    memset(&p.d, 0, sizeof(p.d));
    p.d.mode = GL_TRIANGLES;
    p.d.tri_count = 1;
    d->pass.rasters.push_back(R);
    d->pass.draws.push_back(p);
    d->pass.tris = 1;
    FrameSrc fs{d, &d->pass, 0, HostFrame()};
    Tables t;
    int r = -1;
    if (build_tables(d->x, d->stage, &fs, 1, kTileShiftPlain, true, t) == MTGL_OK)
        r = (int)reinterpret_cast<const DevFrame *>(d->stage.p + t.off_frames)->occlude;
    if ((t.occlude ? 1 : 0) != r) r = -1;
    d->pass.reset();
    mtgl_dev_destroy(d);
    return r;
}
}

namespace mtgl {

size_t scan_temp_words(uint32_t n) { return 2 * (((size_t)n + 2047) / 2048) + 64; }
uint32_t bin_units(uint32_t nrec, int) { return nrec + 31; }
size_t radix_hist_words(uint32_t npairs) { return ((size_t)npairs + 2047) / 2048 * 512 + 64; }

int launch_vertex(const GeomArgs &a, cudaStream_t)
{
    if (a.zero_words) a.rec_total[0] = a.rec_total[1] = 0;
    return say("vertex");
}
int launch_setup_count(const GeomArgs &, cudaStream_t) { return say("count"); }
int launch_setup_emit(const GeomArgs &, cudaStream_t) { return say("emit"); }
int launch_setup_free(const GeomArgs &a, cudaStream_t)
{
    *a.rec_total = g_records;
    return say("setup");
}
int launch_scan(const uint32_t *, uint32_t *, uint32_t, uint32_t *, uint32_t *total_dev, uint32_t *, cudaStream_t,
                const uint32_t *, uint32_t *)
{
    *total_dev = g_records;
    return 1;
}
int launch_bin_count(const BinArgs &a, cudaStream_t)
{
    *a.total_dev = g_pairs;
    if (a.totals_host) {
        a.totals_host[0] = *a.nrec_dev;
        a.totals_host[1] = g_pairs;
    }
    return say("bin");
}
int launch_bin_expand(const BinArgs &, cudaStream_t) { return 1; }
int launch_bin_sort(BinArgs &, cudaStream_t) { return say("sort"); }
int launch_tile_ranges(const BinArgs &, cudaStream_t) { return 1; }
int launch_tile_order(const uint32_t *, uint32_t, uint32_t *, uint32_t *, int, cudaStream_t) { return 2; }
int launch_tile(const TileArgs &a, cudaStream_t)
{
    if (a.guard && (a.guard[0] > a.records_cap || a.guard[1] > a.pairs_cap)) return say("over");
    return say(a.frames[0].host_color ? "tile+read" : "tile");
}
int tile_occupancy(const TileArgs &) { return 4; }
void launch_clear(const ClearOp *, int, FrameDims, uint32_t *, float *, uint8_t *, cudaStream_t) { say("clear"); }
void launch_expand_texels(const uint8_t *, int, int64_t, uint32_t *, cudaStream_t) {}
void launch_mip1(const uint32_t *, int32_t, int32_t, uint32_t *, cudaStream_t) {}
void launch_draw_pixels(const uint32_t *, int32_t, int32_t, int32_t, int32_t, const DevRaster *, FrameDims, uint32_t *,
                        float *, cudaStream_t)
{
}
int launch_readback(const ReadbackItem *, int, int, cudaStream_t) { return 1; }

}  // namespace mtgl
