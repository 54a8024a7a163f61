// The tensor map by which TMA gathers packed 656-byte rows.
#pragma once

#include <cuda.h>

#include "common.cuh"

namespace smla {

constexpr int NO_ROW = 0x7fffffff;             // outside the tensor map: arrives as zeros

// One cache whose rows lie one after the other (pages without padding between them), on a 16-byte boundary: what a tensor map
// needs to name them by their index.
inline bool one_linear_array(const AttnParams& p) {
    return p.layout == SMLA_LAYOUT_V32 && p.extra_topk == 0 && p.block_stride == (int64_t)p.page_block_size * ROW_BYTES &&
           (reinterpret_cast<uintptr_t>(p.kv) & 15u) == 0;
}

// The cache as 32-bit words, 164 per row; boxes of 32 words (128 bytes) of one row, 128B swizzle.  0 or an error code.
int rows_tensor_map(const uint8_t* kv, CUtensorMap* map);

}  // namespace smla
