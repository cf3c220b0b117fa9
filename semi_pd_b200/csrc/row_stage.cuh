// Output rows of a GEMM epilogue through shared memory.  A thread holds one row's columns (its TMEM lane); stored from
// there, a warp's 16-byte stores touch 32 different lines each.  Here a warp stages 64 16-bit (32 fp32) columns of its 32
// rows and writes whole 128-byte pieces of rows.  5172 x 4096 x 512 31.1 -> 26.0 us (a tile's
// epilogue took longer than its eight k-blocks), 4096 x 3648 x 2048 50.5 -> 46.3, 1300 x 6144 x 4096 53.9 -> 52.4.
#pragma once
#include "ptx.cuh"

namespace spd {

constexpr int kStageRow = 144;             // 128 bytes and 16 against bank conflicts
constexpr int kStageWarp = 32 * kStageRow;

// 32 values of this lane's row as T, the first (half 0) or second 32 of 64 columns
template <typename T>
__device__ __forceinline__ void stage_put16(uint8_t* stage, int lane, int half, const float (&v)[32]) {
  uint4* dst = reinterpret_cast<uint4*>(stage + lane * kStageRow + half * 64);
#pragma unroll
  for (int i = 0; i < 4; ++i)
    dst[i] = make_uint4(pack2<T>(v[8 * i], v[8 * i + 1]), pack2<T>(v[8 * i + 2], v[8 * i + 3]),
                        pack2<T>(v[8 * i + 4], v[8 * i + 5]), pack2<T>(v[8 * i + 6], v[8 * i + 7]));
}
// 32 values as fp32 (mode: see f32_result)
template <typename T>
__device__ __forceinline__ void stage_put32(uint8_t* stage, int lane, const float (&v)[32], int mode) {
  float4* dst = reinterpret_cast<float4*>(stage + lane * kStageRow);
#pragma unroll
  for (int i = 0; i < 8; ++i)
    dst[i] = make_float4(f32_result<T>(v[4 * i], mode), f32_result<T>(v[4 * i + 1], mode),
                         f32_result<T>(v[4 * i + 2], mode), f32_result<T>(v[4 * i + 3], mode));
}
// the staged rows to dst (row 0, the first of the staged columns; ld in bytes): rows < `rows`, bytes < `bytes` of a row
__device__ __forceinline__ void stage_out(const uint8_t* stage, int lane, uint8_t* dst, int64_t ld, int rows, int bytes) {
  __syncwarp();
  const int piece = (lane & 7) * 16;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = i * 4 + (lane >> 3);
    if (r < rows && piece < bytes)
      *reinterpret_cast<uint4*>(dst + r * ld + piece) = *reinterpret_cast<const uint4*>(stage + r * kStageRow + piece);
  }
  __syncwarp();  // the next columns may be staged
}

}  // namespace spd
