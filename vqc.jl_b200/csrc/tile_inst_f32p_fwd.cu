// Tile kernels: the FP32 packed body (interpreted form of the compiled passes), forward passes.
#include "tile_kernels_impl.cuh"

template __global__ void vqc::k_tile_packed<9, false>(const __grid_constant__ vqc::TileItem);
template __global__ void vqc::k_tile_packed<10, false>(const __grid_constant__ vqc::TileItem);
template __global__ void vqc::k_tile_packed<11, false>(const __grid_constant__ vqc::TileItem);
template __global__ void vqc::k_tile_packed<12, false>(const __grid_constant__ vqc::TileItem);
