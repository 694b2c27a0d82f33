// Instantiates the tile kernel for C2C and the even real modes together (see
// IO_TILE; one translation unit per instance so the build runs in parallel).
#include "launch_common.cuh"
#include "tile_fft.cuh"

namespace gfft {
int launch_tile_any(const TileArgs& t, int threads, size_t smem, unsigned grid, cudaStream_t st)
{
    static unsigned long long attr_mask = 0;
    auto* k = tile_kernel<kTileMaxThreads, 2, IO_TILE>;
    const cudaError_t e = ensure_smem_attr(k, attr_mask, smem);
    if (e != cudaSuccess) return (int)e;
    return (int)launch_pdl(k, dim3(grid), dim3(threads), smem, st, t);
}
}  // namespace gfft
