// Tile kernels: the classic body, FP64, reverse sweep.
#include "tile_kernels_impl.cuh"

template __global__ void vqc::k_tile<double, true>(const __grid_constant__ vqc::TileItem);
template __global__ void vqc::k_tile_batch<double, true>(const vqc::TileItem*);
