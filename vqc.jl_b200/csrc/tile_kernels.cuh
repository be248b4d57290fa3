// Declarations of the tile kernels (defined in tile_kernels_impl.cuh and
// instantiated in the tile_inst_*.cu translation units, so that the planner
// and the kernels compile in parallel).
#pragma once

#include "tile_plan.cuh"

namespace vqc {

// One pass of one state: the tiles of the pass strided over the grid.
template <class R, bool ADJ>
__global__ void k_tile(const __grid_constant__ TileItem item);
// One pass each of many states (the serving loop): item blockIdx.y.
template <class R, bool ADJ>
__global__ void k_tile_batch(const TileItem* __restrict__ items);
// One pass of one FP32 state on the packed plan, interpreted (the fallback of
// a compiled pass).
template <int M, bool ADJ>
__global__ void k_tile_packed(const __grid_constant__ TileItem item);

}  // namespace vqc
