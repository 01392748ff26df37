// Where the GEMM's activation operand lies in memory, and the tensor map that describes it.  No CUDA types, so that the rule can be run without a GPU.
#pragma once

#include <stddef.h>
#include <stdint.h>

// f16 values as [chunk of 64 values of K][hi, lo][row][64]: a row's piece of a chunk is 128 bytes, the swizzle span.  A box of some rows, both parts and two chunks
// then arrives in the order in which the MMAs want it (per chunk the hi rows, then the lo rows) by a map whose every stride is the one before it times the
// extent of its dimension, as the encoder's description builds them.  Rows of [hi K | lo K] need strides that fall (4 K, 2 K, 128 bytes).
constexpr uint32_t ACT_CHUNK_K = 64, ACT_ROW = ACT_CHUNK_K / 4;

// In units of four values: those of `row` from value 4 * k4 on, the hi part; the lo part lies act_rows_lo behind it, the next row's ACT_ROW.
__host__ __device__ inline size_t act_rows_hi(uint32_t rows, uint32_t row, uint32_t k4) {
  return ((size_t)(k4 / ACT_ROW) * 2 * rows + row) * ACT_ROW + k4 % ACT_ROW;
}
__host__ __device__ inline size_t act_rows_lo(uint32_t rows) { return (size_t)rows * ACT_ROW; }

struct ActMapShape {
  uint64_t dims[4], strides[3];  // value of a chunk, row, part, chunk; bytes
  uint32_t box[4];
  ActMapShape(uint32_t rows, uint32_t K, uint32_t box_rows, uint32_t box_chunks)
      : dims{ACT_CHUNK_K, rows, 2, K / ACT_CHUNK_K}, strides{ACT_CHUNK_K * 2, ACT_CHUNK_K * 2ull * rows, ACT_CHUNK_K * 4ull * rows}, box{ACT_CHUNK_K, box_rows, 2, box_chunks} {}
};
