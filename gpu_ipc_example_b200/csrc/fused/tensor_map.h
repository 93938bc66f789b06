// Tensor map of a row-major 16-bit operand [rows, cols] read in boxes of 64 columns (one 128-byte swizzle row) x
// box_rows rows.
#pragma once

#include <cuda.h>

#include <cstdint>

#include "../common/types.h"

namespace b200ipc {

constexpr int kTileMapCols = 64;

void encode_tile_map(CUtensorMap* map, DType t, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows);

}  // namespace b200ipc
