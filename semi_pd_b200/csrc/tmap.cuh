// Host-side TMA descriptor encoding (implemented in lib.cu).
#pragma once
#include <cuda.h>
#include <stdint.h>

namespace spd {

// A tensor of 16-bit elements in `rank` (at most 5) dimensions, innermost first; strides in elements, from the second
// dimension on.
int make_tmap_sw128(CUtensorMap* out, const void* base, int rank, const uint64_t* dims, const uint64_t* strides,
                    const uint32_t* box);

// 2-D row-major tensor of 16-bit elements [rows, cols] with `row_stride_elems` between rows;
// box = box_rows x box_cols (box_cols * 2 bytes must be 128 for the 128-byte swizzle).
// Out-of-bounds parts of a box are zero-filled by the hardware.
int make_tmap_2d_sw128(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols,
                       uint64_t row_stride_elems, uint32_t box_rows, uint32_t box_cols);

// The same rows as [blocks][rows][64 columns]: one box of box_rows x box_blocks lands as box_blocks consecutive
// swizzle blocks of [box_rows x 128 bytes], with one copy instruction instead of one per block.
int make_tmap_blocks_sw128(CUtensorMap* out, const void* base, uint64_t rows, uint64_t blocks, uint64_t row_stride_elems,
                           uint32_t box_rows, uint32_t box_blocks);

// Cached variant (implemented in gemm.cu): descriptors are pure functions of (pointer, shape,
// box), so steady-state launches do no driver work.  box_cols is fixed at 64 (one swizzle atom).
int get_tmap(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint64_t stride,
             uint32_t box_rows);

}  // namespace spd
