// k_tile.cu — K4 launches: the ordered kernel without deferred colour (k_tile.cuh), and the choice
// between it and the deferred-colour and order-free ones.
#include <atomic>

#include "k_tile.cuh"

namespace mtgl {

int launch_tile(const TileArgs &a, cudaStream_t s)
{
    if (a.ntiles == 0) return 0;
    if (a.order_free) return launch_tile_free(a, s);
    if (a.defer) return launch_tile_deferred(a, s);
    with_tile_kernel<false>(a, [&](auto k, int threads) { launch_tiles(k, a, threads, s); });
    return 1;
}

int tile_occupancy(const TileArgs &a)
{
    // asked on every batch: one answer per kernel, found once (0: not yet)
    static std::atomic<int> known[3][3][4];
    std::atomic<int> &n = known[a.order_free ? 2 : (a.defer ? 1 : 0)][a.tile_shift == 3 ? 0 : (a.tile_shift == 5 ? 2 : 1)]
                               [(a.any_texture ? 1 : 0) + (a.eye_records ? 2 : 0)];
    if (!n.load())
        n.store(a.order_free ? free_per_sm(a)
                : a.defer    ? deferred_per_sm(a)
                             : with_tile_kernel<false>(a, [](auto k, int threads) { return tiles_per_sm(k, threads); }));
    return n.load();
}

}  // namespace mtgl
