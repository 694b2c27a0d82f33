// tile_static.cuh - instantiation of one compile-time tile shape.
#pragma once
#include "launch_common.cuh"
#include "tile_fft.cuh"
#include "tile_list.h"

namespace gfft {

template <int IO, class S>
int launch_tile_shape(const TileArgs& t, int threads, size_t smem, unsigned grid, cudaStream_t st)
{
    static unsigned long long attr_mask = 0;
    auto* k = tile_kernel<kTileMaxThreads, 2, IO, uint32_t, S>;
    const cudaError_t e = ensure_smem_attr(k, attr_mask, smem);
    if (e != cudaSuccess) return (int)e;
    return (int)launch_pdl(k, dim3(grid), dim3(threads), smem, st, t);
}

template <int ID>
struct TileShape;
#define GFFT_SHAPE_R(ID, LL, TT, WW, ...)                   \
    template <>                                             \
    struct TileShape<ID> {                                  \
        using type = TileSpec<LL, TT, WW, true, __VA_ARGS__>; \
    };
#define GFFT_SHAPE_C(ID, LL, TT, WW, ...)                    \
    template <>                                              \
    struct TileShape<ID> {                                   \
        using type = TileSpec<LL, TT, WW, false, __VA_ARGS__>; \
    };
GFFT_TILE_ROWS(GFFT_SHAPE_R)
GFFT_TILE_COLS(GFFT_SHAPE_C)
#undef GFFT_SHAPE_R
#undef GFFT_SHAPE_C

template <int ID>
int launch_tile_id(int io, const TileArgs& t, int threads, size_t smem, unsigned grid, cudaStream_t st)
{
    using S = typename TileShape<ID>::type;
    if (io == IO_C2C) return launch_tile_shape<IO_C2C, S>(t, threads, smem, grid, st);
    // long real passes pair columns in tiles of 16 (R2C, 8 from 1024 points)
    // and 8 (C2R)
    constexpr bool r2c = S::ROWS || S::W == 16 || S::L == 1024, c2r = S::ROWS || S::W == 8;
    if constexpr (r2c) {
        if (io == IO_R2C_EVEN) return launch_tile_shape<IO_R2C_EVEN, S>(t, threads, smem, grid, st);
    }
    if constexpr (c2r) {
        if (io == IO_C2R_EVEN) return launch_tile_shape<IO_C2R_EVEN, S>(t, threads, smem, grid, st);
    }
    return kNoTileShape;
}

}  // namespace gfft

#define GFFT_TILE_TU(ID)                                                                                        \
    namespace gfft {                                                                                            \
    int launch_tile_s##ID(int io, const TileArgs& t, int threads, size_t smem, unsigned grid, cudaStream_t st)   \
    {                                                                                                           \
        return launch_tile_id<ID>(io, t, threads, smem, grid, st);                                              \
    }                                                                                                           \
    }
