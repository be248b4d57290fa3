// Tile kernels: the classic body, FP64, forward passes.
#include "tile_kernels_impl.cuh"

template __global__ void vqc::k_tile<double, false>(const __grid_constant__ vqc::TileItem);
template __global__ void vqc::k_tile_batch<double, false>(const vqc::TileItem*);
