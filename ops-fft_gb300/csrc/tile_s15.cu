// tile shape 15 of tile_list.h
#include "tile_static.cuh"

GFFT_TILE_TU(15)
