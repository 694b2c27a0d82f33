// tile_fft.cu - launchers of the tile kernel (instances in tile_io*.cu).
#include <initializer_list>

#include "launch_common.cuh"
#include "tile_fft.cuh"
#include "tile_list.h"

namespace gfft {
int launch_tile_any(const TileArgs& t, int threads, size_t smem, unsigned grid, cudaStream_t st);
int launch_tile_io0(const TileArgs& t, int threads, size_t smem, unsigned grid, cudaStream_t st);
int launch_tile_io0w(const TileArgs& t, int threads, size_t smem, unsigned grid, cudaStream_t st);
int launch_tile_io1(const TileArgs& t, int threads, size_t smem, unsigned grid, cudaStream_t st);
int launch_tile_io2(const TileArgs& t, int threads, size_t smem, unsigned grid, cudaStream_t st);
int launch_tile_io3(const TileArgs& t, int threads, size_t smem, unsigned grid, cudaStream_t st);
int launch_tile_io4(const TileArgs& t, int threads, size_t smem, unsigned grid, cudaStream_t st);

#define GFFT_DECL_SHAPE(ID, ...) \
    int launch_tile_s##ID(int io, const TileArgs& t, int threads, size_t smem, unsigned grid, cudaStream_t st);
GFFT_TILE_ROWS(GFFT_DECL_SHAPE)
GFFT_TILE_COLS(GFFT_DECL_SHAPE)
#undef GFFT_DECL_SHAPE

namespace {

// Whether a launch's tile is the compile-time shape L, T, W, radices.
bool shape_is(const TileArgs& t, int L, int T, int W, bool rows, std::initializer_list<int> rad)
{
    if (t.ip.L != L || t.ip.nthr != T || t.W != W || (t.rows != 0) != rows || t.ip.npass != (int)rad.size()) return false;
    int p = 0;
    for (int r : rad)
        if (t.ip.pass[p++].radix != r) return false;
    int k = 0;  // the shared padding that goes with them
    while ((1 << k) < *rad.begin()) ++k;
    return t.pshift == (rad.size() > 1 && (1 << k) == *rad.begin() ? k : 30);
}

int launch_tile(int io, const TileArgs& t, size_t smem, bool shared, cudaStream_t st)
{
    int threads = t.W * t.ip.nthr;
    threads = (threads + 31) & ~31;
    if (t.W < 1 || t.ip.nthr < 1 || threads > kTileMaxThreads || t.ncols == 0 || smem > (size_t)kMaxSmemBytes)
        return (int)cudaErrorInvalidValue;
    const unsigned per = t.rows || !t.M ? (unsigned)t.W : (unsigned)t.W / 2;  // paired columns: two per unit
    if (per < 1) return (int)cudaErrorInvalidValue;
    const unsigned grid = (t.ncols + per - 1) / per;
    const bool wide = (int64_t)t.ip.L * (t.in_st8 > t.out_st8 ? t.in_st8 : t.out_st8) > 0xffffffffll;
    if (!wide && (io == IO_C2C || io == IO_R2C_EVEN || io == IO_C2R_EVEN)) {
        int rc = kNoTileShape;
#define GFFT_SHAPE_ROW(ID, LL, TT, WW, ...) \
    if (shape_is(t, LL, TT, WW, true, {__VA_ARGS__})) rc = launch_tile_s##ID(io, t, threads, smem, grid, st);
#define GFFT_SHAPE_COL(ID, LL, TT, WW, ...) \
    if (shape_is(t, LL, TT, WW, false, {__VA_ARGS__})) rc = launch_tile_s##ID(io, t, threads, smem, grid, st);
        GFFT_TILE_ROWS(GFFT_SHAPE_ROW)
        GFFT_TILE_COLS(GFFT_SHAPE_COL)
#undef GFFT_SHAPE_ROW
#undef GFFT_SHAPE_COL
        if (rc != kNoTileShape) return rc;
    }
    if (shared && !wide && (io == IO_C2C || io == IO_R2C_EVEN || io == IO_C2R_EVEN))
        return launch_tile_any(t, threads, smem, grid, st);
    switch (io) {
    case IO_C2C:
        // the span of one transform decides the offset width
        if (wide) return launch_tile_io0w(t, threads, smem, grid, st);
        return launch_tile_io0(t, threads, smem, grid, st);
    case IO_R2C_EVEN: return launch_tile_io1(t, threads, smem, grid, st);
    case IO_C2R_EVEN: return launch_tile_io2(t, threads, smem, grid, st);
    case IO_R2C_ODD: return launch_tile_io3(t, threads, smem, grid, st);
    case IO_C2R_ODD: return launch_tile_io4(t, threads, smem, grid, st);
    default: return (int)cudaErrorInvalidValue;
    }
}

constexpr int64_t kTileMaxCols = (int64_t(1) << 31) - 64;  // 32-bit column arithmetic

}  // namespace
}  // namespace gfft

using namespace gfft;

extern "C" int gfft_launch_tile_row(const RowArgs* a, void* stream)
{
    if (a->ntf < 1 || a->ntf > kTileMaxCols) return (int)cudaErrorInvalidValue;
    TileArgs t{};
    t.ip = a->ip;
    t.tw = static_cast<const float2*>(a->tw);
    t.post = static_cast<const float2*>(a->post_tw);
    t.in = a->in;
    t.out = a->out;
    t.ncols = (uint32_t)a->ntf;
    t.cpi = t.in_split = t.out_split = t.tw_div = t.ons = tile_div(1);
    t.T = tile_div(a->ip.nthr);
    t.in_dist = a->in_dist;
    t.out_dist = a->out_dist;
    t.in_st8 = t.out_st8 = 8;
    t.W = a->tfpc;
    t.rows = 1;
    t.emul = 1;
    t.cmul = a->lpad;
    t.pshift = a->pshift;
    t.conj_in = a->conj_in;
    t.conj_out = a->conj_out;
    t.weight = a->weight;
    t.scale = a->scale;
    t.wl = a->wload;
    t.wdist = a->wdist;
    t.io = a->io_mode;
    return launch_tile(a->io_mode, t, (size_t)a->smem_bytes, a->tile == 2, static_cast<cudaStream_t>(stream));
}

extern "C" int gfft_launch_tile_col(const ColArgs* a, void* stream)
{
    if (a->ncols < 1 || a->ncols > kTileMaxCols) return (int)cudaErrorInvalidValue;
    TileArgs t{};
    t.ip = a->ip;
    t.tw = static_cast<const float2*>(a->tw);
    if (a->ons > 1) {
        if (a->otw2d) {
            t.otw = static_cast<const float2*>(a->otw_hi);
            t.otw_lo = static_cast<const float2*>(a->otw_lo);
        } else {
            t.otw_hi = static_cast<const float2*>(a->otw_hi);
            t.otw_lo = static_cast<const float2*>(a->otw_lo);
        }
    }
    t.otw_shift = a->otw_shift;
    t.in = a->in;
    t.out = a->out;
    t.ncols = (uint32_t)a->ncols;
    // a split at or beyond the columns of an item never divides
    t.cpi = tile_div(a->cpi);
    t.in_split = tile_div(a->in_split < a->cpi ? a->in_split : a->cpi);
    t.out_split = tile_div(a->out_split < a->cpi ? a->out_split : a->cpi);
    t.tw_div = tile_div(a->tw_div < a->cpi ? a->tw_div : a->cpi);
    t.ons = tile_div(a->ons);
    t.T = tile_div(a->ip.nthr);
    t.in_dist = a->in_dist;
    t.in_hi = a->in_hi;
    t.in_lo = a->in_lo;
    t.in_st8 = 8 * a->in_stride;
    t.out_dist = a->out_dist;
    t.out_hi = a->out_hi;
    t.out_lo = a->out_lo;
    t.out_st8 = 8 * a->out_stride;
    t.W = a->tfpc;
    while ((1 << t.wshift) < t.W) ++t.wshift;
    if ((1 << t.wshift) != t.W) return (int)cudaErrorInvalidValue;
    t.rows = 0;
    t.emul = a->tfpc;
    t.cmul = 1;
    t.pshift = a->pshift;
    t.staged_out = a->staged_out;
    t.spitch = a->spitch;
    t.conj_in = a->conj_in;
    t.conj_out = a->conj_out;
    t.scale = a->scale;
    if (a->io_mode != IO_C2C) {
        t.M = (uint32_t)a->pair_m;
        t.post = static_cast<const float2*>(a->post_tw);
        t.weight = a->weight;
        if (t.M < 1 || !t.post) return (int)cudaErrorInvalidValue;
    }
    t.io = a->io_mode;
    return launch_tile(a->io_mode, t, (size_t)a->smem_bytes, a->tile == 2, static_cast<cudaStream_t>(stream));
}
