// tile_list.h - the tiles that are compiled with their length, threads and
// radices as constants (csrc/tile_fft.cuh): divisions, padding and strides
// become immediates, and a quarter fewer instructions remain (us, constants /
// arguments: C2C rows 512 x 32768 43.4 / 46.9, 4096 x 4096 44.0 / 51.3, one row
// of 1024 points 2.0 / 3.5, R2C 8192 x 4096 54.1 / 65.8, 262144 x 128 123 / 151,
// C2C 1048576 x 32 237 / 274, columns 512 x 65536 93 / 109).
// X(id, L, T, W, radices...): rows for C2C and the even real modes, columns
// for C2C and the pairs of the long even real passes.  The launcher takes a
// shape whenever a plan's tile equals it and the argument-driven kernel for
// every other tile.  Shapes with twice the threads serve few rows.  Each is a translation unit of its own (tile_s<id>.cu) so
// the build runs in parallel.
#pragma once
namespace gfft {
constexpr int kNoTileShape = -1;  // the shape has no instance of this mode
}
#define GFFT_TILE_ROWS(X)            \
    X(0, 512, 32, 2, 8, 8, 8)        \
    X(1, 1024, 64, 1, 16, 8, 8)      \
    X(2, 1500, 150, 1, 15, 10, 10)   \
    X(3, 2048, 128, 1, 16, 16, 8)    \
    X(4, 4096, 256, 1, 16, 16, 16)   \
    X(5, 128, 8, 8, 16, 8)           \
    X(6, 256, 16, 4, 16, 16)         \
    X(7, 8192, 512, 1, 16, 8, 8, 8)  \
    X(15, 512, 64, 1, 8, 8, 8)       \
    X(16, 1024, 128, 1, 16, 8, 8)    \
    X(17, 2048, 256, 1, 16, 16, 8)   \
    X(18, 128, 16, 4, 16, 8)
#define GFFT_TILE_COLS(X)            \
    X(8, 128, 8, 16, 16, 8)          \
    X(9, 256, 16, 8, 16, 16)         \
    X(10, 256, 16, 16, 16, 16)       \
    X(11, 512, 32, 8, 8, 8, 8)       \
    X(12, 512, 32, 16, 8, 8, 8)      \
    X(13, 1024, 64, 8, 16, 8, 8)     \
    X(14, 2048, 128, 4, 16, 16, 8)
