// Tensor maps of the TMA loads (host side).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace fmoe {

// Row-major [outer, inner] matrix of 16-bit elements (dtype as in DType), 128-byte swizzle (64-byte
// where a box is 32 columns wide).  False when the driver refuses the map.
bool make_map_2d(CUtensorMap* map, int dtype, const void* base, uint64_t inner, uint64_t outer, uint32_t box_inner,
                 uint32_t box_outer);

// Row-major [outer, mid, inner], boxes of one matrix: rows past `mid` are filled with zeros.
bool make_map_3d(CUtensorMap* map, int dtype, const void* base, uint64_t inner, uint64_t mid, uint64_t outer,
                 uint32_t box_inner, uint32_t box_mid);

// Row-major [outer, inner] seen as blocks of 64 columns (inner a multiple of 64): coordinates are (0,
// row, block), a box is `box_blocks` blocks of [box_outer, 64], one behind the other.
bool make_map_columns(CUtensorMap* map, int dtype, const void* base, uint64_t inner, uint64_t outer, uint32_t box_outer,
                      uint32_t box_blocks);

}  // namespace fmoe
