// Tile kernels: the FP32 packed body (interpreted form of the compiled passes), reverse sweep.
#include "tile_kernels_impl.cuh"

template __global__ void vqc::k_tile_packed<9, true>(const __grid_constant__ vqc::TileItem);
template __global__ void vqc::k_tile_packed<10, true>(const __grid_constant__ vqc::TileItem);
template __global__ void vqc::k_tile_packed<11, true>(const __grid_constant__ vqc::TileItem);
template __global__ void vqc::k_tile_packed<12, true>(const __grid_constant__ vqc::TileItem);
