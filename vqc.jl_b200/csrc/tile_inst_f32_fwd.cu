// Tile kernels: the classic body, FP32, forward passes.
#include "tile_kernels_impl.cuh"

template __global__ void vqc::k_tile<float, false>(const __grid_constant__ vqc::TileItem);
template __global__ void vqc::k_tile_batch<float, false>(const vqc::TileItem*);
