// tile shape 13 of tile_list.h
#include "tile_static.cuh"

GFFT_TILE_TU(13)
