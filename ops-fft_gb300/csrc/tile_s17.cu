// tile shape 17 of tile_list.h
#include "tile_static.cuh"

GFFT_TILE_TU(17)
