// Tile metadata left by the tile stage (tiles.cu), read by the coverage
// kernels, the span scan and the differentiable stages.
#pragma once

#include "common.cuh"
#include "internal.h"

namespace ochre {

// Tile metadata, three words per tile: the first bin entry of the tile in
// the sorted entries (its bins run to the next tile's first, crossing entries
// between), its tile coordinates, and its raster with two flags.
constexpr uint32_t RF_RASTER = MAX_RASTERS - 1u;
constexpr uint32_t RF_WIND = 1u << 30;   // the crossings of its raster sorted before it sum to a nonzero winding
constexpr uint32_t RF_ROW = 1u << 31;    // it starts its (raster, tile_y) row
__device__ __forceinline__ uint32_t pack_tile(int tx, int ty) {
    return (uint32_t)(uint16_t)(int16_t)tx | ((uint32_t)(uint16_t)(int16_t)ty << 16);
}
__device__ __forceinline__ int tile_tx(uint32_t xy) { return (int)(int16_t)(xy & 0xffffu); }
__device__ __forceinline__ int tile_ty(uint32_t xy) { return (int)(int16_t)(xy >> 16); }
struct TileView {
    const uint32_t* head;
    const uint32_t* xy;
    const uint32_t* rf;
    uint32_t n_entries;          // sorted entries: the end of the last tile's bins
    const uint32_t* entries_dev; // the same held on the device (graph replays), else null
    __device__ __forceinline__ uint32_t end() const { return (uint32_t)dev_count(n_entries, entries_dev); }
};

}  // namespace ochre
