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
