// TMA tensor maps of row-major matrices.
#pragma once

#include <cuda.h>

#include "common.cuh"

namespace cera {

// [rows][ld] elements of elem_bytes (ld * elem_bytes a multiple of 16), boxes of box_cols x box_rows elements; elements outside
// read as zero.
int32_t tensor_map_2d(CUtensorMap *map, CUtensorMapDataType type, uint32_t elem_bytes, const void *base, uint64_t rows, uint64_t ld, uint32_t box_cols,
                      uint32_t box_rows, CUtensorMapSwizzle swizzle, CUtensorMapL2promotion promotion);

// bf16, boxes laid down with the 128-byte swizzle (box_cols = 64).
inline int32_t tensor_map_bf16(CUtensorMap *map, const void *base, uint64_t rows, uint64_t ld, uint32_t box_cols, uint32_t box_rows) {
    return tensor_map_2d(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base, rows, ld, box_cols, box_rows, CU_TENSOR_MAP_SWIZZLE_128B,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
}

}  // namespace cera
