// k_tile_defer.cu — K4 launches with deferred colour (the kernel is in k_tile.cuh; the halves
// compile in parallel).
#include "k_tile.cuh"

namespace mtgl {

int launch_tile_deferred(const TileArgs &a, cudaStream_t s)
{
    with_tile_kernel<true>(a, [&](auto k, int threads) { launch_tiles(k, a, threads, s); });
    return 1;
}

int deferred_per_sm(const TileArgs &a)
{
    return with_tile_kernel<true>(a, [](auto k, int threads) { return tiles_per_sm(k, threads); });
}

}  // namespace mtgl
