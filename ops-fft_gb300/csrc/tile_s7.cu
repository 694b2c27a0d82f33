// tile shape 7 of tile_list.h
#include "tile_static.cuh"

GFFT_TILE_TU(7)
