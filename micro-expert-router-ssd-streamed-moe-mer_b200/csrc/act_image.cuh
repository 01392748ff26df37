// Activation rows as the streaming kernels multiply them, prepared once per row: mma.sync B fragments and zero-point terms in
// global memory, from where a CTA fetches the part of a token pass that it needs by bulk copies.
//
// A row of K values becomes K / 32 records of 64 bytes of f16 hi parts, as many of lo parts, and two runs of K / 32 fp32 terms
// (hi and lo of -zp * 2^-24 * sum of the block), after an exact power-of-two scaling of the row.
// Built by whoever has the row at hand (router, grouping, SiLU tail).  Every CTA that touched one of a token's experts used to build the
// fragments itself, 3 to 5 us each time with its sixteen warps waiting at barriers.
#pragma once

#include <cuda_fp16.h>
#include <stdint.h>

#include "../../include/mer_b200.h"
#include "decode.cuh"
#include "kernels.h"

namespace {

// Position of block element j in the per-block fragment order, and the extra exact scale of that slot (Q4_0 high nibbles
// sit 4 mantissa bits higher, so their activations carry 2^-4).
__device__ __forceinline__ void frag_slot(int dtype, uint32_t j, uint32_t &pos, float &slot_scale) {
  const bool q4 = dtype == MER_DTYPE_Q4_0;
  const uint32_t hi = q4 ? j >> 4 : (j & 7u) >> 2, t = q4 ? (j & 15u) >> 2 : j >> 3, e = j & 3u;
  // thread t order: [+0, +2, +1, +3 | the same of the second half]
  const uint32_t within = (e == 0) ? 0 : (e == 2) ? 1 : (e == 1) ? 2 : 3;
  pos = t * 8 + hi * 4 + within;
  slot_scale = q4 && hi ? 0.0625f : 1.0f;
}

// Four scaled values, number `q` of their row's groups of four; eight consecutive lanes hold a block and all lanes of the warp call.
__device__ __forceinline__ void image_store4(int dtype, float4 v, uint32_t q, bool inside, uint8_t *hi_row, uint8_t *lo_row, float *seed_hi, float *seed_lo) {
  const uint32_t kb = q >> 3;
  uint32_t pos;
  float ss;
  frag_slot(dtype, (q & 7u) * 4, pos, ss);  // the four elements land at pos + {0, 2, 1, 3}
  const __half2 h0 = __floats2half2_rn(v.x * ss, v.z * ss), h1 = __floats2half2_rn(v.y * ss, v.w * ss);
  const float2 f0 = __half22float2(h0), f1 = __half22float2(h1);
  const __half2 l0 = __floats2half2_rn(v.x * ss - f0.x, v.z * ss - f0.y), l1 = __floats2half2_rn(v.y * ss - f1.x, v.w * ss - f1.y);
  if (inside) {
    *reinterpret_cast<uint2 *>(hi_row + (size_t)kb * 64 + pos * 2) = make_uint2(h2_bits(h0), h2_bits(h1));
    *reinterpret_cast<uint2 *>(lo_row + (size_t)kb * 64 + pos * 2) = make_uint2(h2_bits(l0), h2_bits(l1));
  }
  float sum = (v.x + v.y) + (v.z + v.w);
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if (inside && (q & 7u) == 0) {
    const float zp = dtype == MER_DTYPE_Q4_0 ? 8.0f : 128.0f, seed = -zp * sum * (1.0f / POW2_24), hi = tf32_round(seed);
    seed_hi[kb] = hi, seed_lo[kb] = tf32_round(seed - hi);
  }
}

// Where row `i` of the activations of width K lies: `rows` = f16 parts, `seeds` = zero-point terms.
struct ImageRow {
  uint8_t *hi, *lo;
  float *seed_hi, *seed_lo;
  __device__ ImageRow(void *rows, float *seeds, size_t i, uint32_t K) {
    hi = static_cast<uint8_t *>(rows) + i * K * 4, lo = hi + (size_t)K * 2;
    const uint32_t kb4 = image_seed_stride(K);
    seed_hi = seeds + i * 2 * kb4, seed_lo = seed_hi + kb4;
  }
};

// Row `token` of d.x by one CTA of `threads` threads (whole warps, at most 32 of them).  What bounds it is latency: the loads of four steps are
// in flight together, and the second pass finds the row in L1.
__device__ __forceinline__ void build_x_image(const MoeDispatch &d, uint32_t token, uint32_t tid, uint32_t threads, float *s_max) {
  constexpr int BATCH = 4;
  const uint32_t K = d.D, n4 = K / 4, limit = (n4 + 31) & ~31u;
  const float4 *src = reinterpret_cast<const float4 *>(d.x + (size_t)token * K);
  float mx = 0.0f;
#pragma unroll 1
  for (uint32_t i0 = tid; i0 < n4; i0 += BATCH * threads) {
    float4 v[BATCH];
#pragma unroll
    for (int u = 0; u < BATCH; u++) v[u] = i0 + u * threads < n4 ? __ldg(src + i0 + u * threads) : make_float4(0, 0, 0, 0);
#pragma unroll
    for (int u = 0; u < BATCH; u++) mx = nan_max(nan_max(nan_max(nan_max(mx, fabsf(v[u].x)), fabsf(v[u].y)), fabsf(v[u].z)), fabsf(v[u].w));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = nan_max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((tid & 31) == 0) s_max[tid >> 5] = mx;
  __syncthreads();
  mx = 0.0f;
#pragma unroll 1
  for (uint32_t w = 0; w < threads / 32; w++) mx = nan_max(mx, s_max[w]);
  float sc = 1.0f;
  if (mx > 0.0f && isfinite(mx)) {
    int e;
    frexpf(mx, &e);              // mx = m * 2^e, m in [0.5, 1)
    sc = ldexpf(1.0f, 9 - e);    // mx * sc in [256, 512)
  } else if (mx != mx || isinf(mx)) {
    sc = mx;  // non-finite activations poison the row, as they would in fp32
  }
  if (tid == 0) d.x_un[token] = POW2_24 / sc;
  const ImageRow row(d.x_rows, d.act_seeds, token, K);
#pragma unroll 1
  for (uint32_t i0 = tid; i0 < limit; i0 += BATCH * threads) {
    float4 v[BATCH];
#pragma unroll
    for (int u = 0; u < BATCH; u++) v[u] = i0 + u * threads < n4 ? __ldg(src + i0 + u * threads) : make_float4(0, 0, 0, 0);
#pragma unroll
    for (int u = 0; u < BATCH; u++) {
      const uint32_t q = i0 + u * threads;
      if (q >= limit) break;  // uniform in a warp
      v[u].x *= sc, v[u].y *= sc, v[u].z *= sc, v[u].w *= sc;  // exact (power of two) unless it overflows
      image_store4(d.dtype, v[u], q, q < n4, row.hi, row.lo, row.seed_hi, row.seed_lo);
    }
  }
}
// The same by a CTA of 256 threads for a token that may have none of its experts here (expert parallelism).
__device__ __forceinline__ void build_wanted_image(const MoeDispatch &d, uint32_t token, float *s_max) {
  bool wanted = false;
  for (uint32_t i = threadIdx.x; i < d.slots; i += 256) wanted |= d.pair_expert[(size_t)token * d.slots + i] != MER_NONE;
  if (__syncthreads_or(wanted)) build_x_image(d, token, threadIdx.x, 256, s_max);
}

}  // namespace
