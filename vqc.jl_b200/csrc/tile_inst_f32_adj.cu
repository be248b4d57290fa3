// Tile kernels: the classic body, FP32, reverse sweep.
#include "tile_kernels_impl.cuh"

template __global__ void vqc::k_tile<float, true>(const __grid_constant__ vqc::TileItem);
template __global__ void vqc::k_tile_batch<float, true>(const vqc::TileItem*);
