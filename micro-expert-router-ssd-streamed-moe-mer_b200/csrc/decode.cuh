// Device helpers shared by the decode kernels (kernels_stream.cu, kernels_flat.cu): integer weights as f16 subnormals, mma.sync.
// (kernels_gemm.cu: h2_bits.)
#pragma once

#include <cuda_fp16.h>
#include <stdint.h>

namespace {

constexpr float POW2_24 = 16777216.0f;

// D = A * B + C with separate C so that a seed / zero needs no register moves.
__device__ __forceinline__ void mma_f16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                        uint32_t b1, float c0, float c1, float c2, float c3) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(c0), "f"(c1), "f"(c2), "f"(c3));
}
// D += A * B, A [16 x 4] and B [4 x 8] in tf32.
__device__ __forceinline__ void mma_tf32(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm("mma.sync.aligned.m16n8k4.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(b0));
}
__device__ __forceinline__ float tf32_round(float v) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(v));
  return __uint_as_float(r);
}
__device__ __forceinline__ float nan_max(float a, float b) { return (b > a || b != b) ? b : a; }  // NaN sticks


// Eight weights of one row slot of one block -> four f16x2 registers holding the integer fields as
// subnormals: {MMA0.k(2t,2t+1), MMA0.k(2t+8,2t+9), MMA1.k(2t,2t+1), MMA1.k(2t+8,2t+9)}.
__device__ __forceinline__ void unpack_q4(uint32_t v, uint32_t (&r)[4]) {
  const uint32_t v8 = v >> 8;
  r[0] = v & 0x000F000Fu;   // low nibbles of bytes 0, 2  -> elements 4t, 4t+2
  r[1] = v8 & 0x000F000Fu;  // low nibbles of bytes 1, 3  -> elements 4t+1, 4t+3
  r[2] = v & 0x00F000F0u;   // high nibbles -> elements 16 + ... (x16, undone on the activation side)
  r[3] = v8 & 0x00F000F0u;
}
__device__ __forceinline__ void unpack_q8(uint32_t lo, uint32_t hi, uint32_t (&r)[4]) {
  // int8 -> biased unsigned byte (q + 128) in the low mantissa bits
  r[0] = (lo ^ 0x80808080u) & 0x00FF00FFu;
  r[1] = ((lo >> 8) ^ 0x00808080u) & 0x00FF00FFu;
  r[2] = (hi ^ 0x80808080u) & 0x00FF00FFu;
  r[3] = ((hi >> 8) ^ 0x00808080u) & 0x00FF00FFu;
}
// The same for bytes that are stored as q + 128 (layout.cuh): four instructions for eight weights instead of six.
__device__ __forceinline__ void unpack_q8_biased(uint32_t lo, uint32_t hi, uint32_t (&r)[4]) {
  r[0] = lo & 0x00FF00FFu, r[1] = __byte_perm(lo, 0u, 0x4341);
  r[2] = hi & 0x00FF00FFu, r[3] = __byte_perm(hi, 0u, 0x4341);
}
__device__ __forceinline__ float2 h2_to_f2(uint32_t v) { return __half22float2(*reinterpret_cast<const __half2 *>(&v)); }

__device__ __forceinline__ uint32_t h2_bits(__half2 v) { return *reinterpret_cast<uint32_t *>(&v); }
}  // namespace
