// Router logits of a few hundred tokens and more: logits[t][e] = x[t] . w[e], on the tensor cores at no less than fp32 precision.
//
//   * Both operands are split into f16 hi + lo parts after exact power-of-two scalings: a router row by its maximum when the router is
//     installed, a token's 64 values at a time by theirs.  Three products (hi*hi, hi*lo, lo*hi) of a chunk of 64 values are summed in the
//     tensor core, 12 additions, and the chunk's sum is unscaled and added in fp32: the tensor core's additions round towards zero, and a
//     whole row of 7168 values summed there would be off by 1e-5.  Measured against 64 bits: profiles of the error in the launch rule.
//   * The router's parts lie in mma.sync B fragment order, K permuted within every 16 values so that a lane's four are neighbours in
//     memory: a chunk of an expert tile is one bulk copy, a fragment one 128-bit load.  A fragments are made in registers from the rows of x.
//   * A CTA computes 128 tokens (16 per warp) x 8 NTN experts over a slice of K; k_router adds the slices.
// What bounds it: the legacy tensor path, 8 cycles per m16n8k16 and scheduler.  4096 tokens x 256 experts x 7168: see launch_router_logits.
#include "kernels.h"

#include <cuda_fp16.h>

#include <algorithm>

#include "../../include/mer_b200.h"
#include "decode.cuh"
#include "ptx.cuh"

namespace {

constexpr uint32_t LG_WARPS = 8, LG_THREADS = LG_WARPS * 32, LG_TOKENS = LG_WARPS * 16;
constexpr uint32_t CHUNK = 64, STEPS = CHUNK / 16;  // values of K per stage; MMA steps
constexpr uint32_t FRAG = 512;                      // bytes of one expert tile's fragments of one step: 32 lanes x {hi 2 x f16x2, lo 2 x f16x2}
constexpr uint32_t TILE_CHUNK = STEPS * FRAG;
constexpr uint32_t STAGES = 4;

__device__ __forceinline__ float pow2_scale(float mx) {  // mx * scale in [256, 512); 1 for zero and non-finite rows
  if (!(mx > 0.0f) || !isfinite(mx)) return 1.0f;
  int e;
  frexpf(mx, &e);
  return ldexpf(1.0f, max(-100, min(100, 9 - e)));
}

// One router row per CTA -> its fragments, and 1 / scale.  Rows past the last expert are zeros.
__global__ void __launch_bounds__(256) k_split_router(const float *__restrict__ w, uint32_t E, uint32_t D, uint8_t *__restrict__ out, float *__restrict__ unscale) {
  __shared__ float s_max[8];
  const uint32_t e = blockIdx.x, n_tiles = gridDim.x / 8;
  float mx = 0.0f;
  if (e < E)
    for (uint32_t k = threadIdx.x; k < D; k += 256) mx = fmaxf(mx, fabsf(w[(size_t)e * D + k]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = mx;
  __syncthreads();
  for (int i = 0; i < 8; i++) mx = fmaxf(mx, s_max[i]);
  const float sc = pow2_scale(mx);
  if (threadIdx.x == 0) unscale[e] = 1.0f / sc;
  for (uint32_t k = threadIdx.x; k < D; k += 256) {
    const float v = e < E ? w[(size_t)e * D + k] * sc : 0.0f;
    const __half hi = __float2half_rn(v), lo = __float2half_rn(v - __half2float(hi));
    const uint32_t kk = k % 16, lane = (e % 8) * 4 + kk / 4;
    __half *dst = reinterpret_cast<__half *>(out + ((size_t)(k / CHUNK) * n_tiles + e / 8) * TILE_CHUNK + k % CHUNK / 16 * FRAG + lane * 16);
    dst[kk % 4] = hi, dst[4 + kk % 4] = lo;
  }
}

__device__ __forceinline__ void mma_acc(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) { mma_f16(d, a[0], a[1], a[2], a[3], b0, b1, d[0], d[1], d[2], d[3]); }
__device__ __forceinline__ float max4(float m, float4 v) { return nan_max(nan_max(nan_max(nan_max(m, fabsf(v.x)), fabsf(v.y)), fabsf(v.z)), fabsf(v.w)); }
// Four neighbouring values of a row -> its two A registers, hi and lo.
__device__ __forceinline__ void split4(float4 v, float sc, uint32_t &h0, uint32_t &h1, uint32_t &l0, uint32_t &l1) {
  v.x *= sc, v.y *= sc, v.z *= sc, v.w *= sc;  // exact
  const __half2 a = __floats2half2_rn(v.x, v.y), b = __floats2half2_rn(v.z, v.w);
  const float2 fa = __half22float2(a), fb = __half22float2(b);
  h0 = h2_bits(a), h1 = h2_bits(b);
  l0 = h2_bits(__floats2half2_rn(v.x - fa.x, v.y - fa.y)), l1 = h2_bits(__floats2half2_rn(v.z - fb.x, v.w - fb.y));
}

template <int NTN>
__global__ void __launch_bounds__(LG_THREADS, 1) k_router_logits(const __grid_constant__ RouterDev r, const float *__restrict__ x, uint32_t T, uint32_t D, uint32_t ksplit,
                                                                 float *__restrict__ logits, uint32_t *status) {
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ uint64_t full[STAGES];
  constexpr uint32_t STAGE = NTN * TILE_CHUNK;
  const uint32_t E = r.num_experts, n_tiles = (E + 7) / 8, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const uint32_t nt0 = blockIdx.x * NTN, nt = min((uint32_t)NTN, n_tiles - nt0);
  const uint32_t n_chunks = D / CHUNK / ksplit, c0 = blockIdx.z * n_chunks;
  const uint32_t row0 = blockIdx.y * LG_TOKENS + warp * 16 + g, row1 = row0 + 8;
  const float4 *x0 = reinterpret_cast<const float4 *>(x + (size_t)min(row0, T - 1) * D) + t, *x1 = reinterpret_cast<const float4 *>(x + (size_t)min(row1, T - 1) * D) + t;
  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < STAGES; s++) mbar_init(&full[s], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  auto issue = [&](uint32_t c) {  // chunk c of the slice into its stage, by one thread
    uint64_t *bar = &full[c % STAGES];
    mbar_expect_tx(bar, nt * TILE_CHUNK);
    bulk_g2s(smem + c % STAGES * STAGE, r.w_split + ((size_t)(c0 + c) * n_tiles + nt0) * TILE_CHUNK, nt * TILE_CHUNK, bar);
  };
  if (threadIdx.x == 0)
    for (uint32_t c = 0; c < min(STAGES, n_chunks); c++) issue(c);
  float4 v0[STEPS], v1[STEPS];
  auto load = [&](uint32_t c) {
#pragma unroll
    for (uint32_t s = 0; s < STEPS; s++) v0[s] = __ldg(x0 + (c0 + c) * (CHUNK / 4) + s * 4), v1[s] = __ldg(x1 + (c0 + c) * (CHUNK / 4) + s * 4);
  };
  load(0);
  float sum[NTN][4];
#pragma unroll
  for (int n = 0; n < NTN; n++) sum[n][0] = sum[n][1] = sum[n][2] = sum[n][3] = 0.0f;
  bool ok = true;
#pragma unroll 1
  for (uint32_t c = 0; c < n_chunks; c++) {
    float m0 = 0.0f, m1 = 0.0f;
#pragma unroll
    for (uint32_t s = 0; s < STEPS; s++) m0 = max4(m0, v0[s]), m1 = max4(m1, v1[s]);
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) m0 = nan_max(m0, __shfl_xor_sync(0xffffffffu, m0, o)), m1 = nan_max(m1, __shfl_xor_sync(0xffffffffu, m1, o));
    const float s0 = pow2_scale(m0), s1 = pow2_scale(m1), u0 = 1.0f / s0, u1 = 1.0f / s1;
    uint32_t ah[STEPS][4], al[STEPS][4];
#pragma unroll
    for (uint32_t s = 0; s < STEPS; s++) {
      split4(v0[s], s0, ah[s][0], ah[s][2], al[s][0], al[s][2]);
      split4(v1[s], s1, ah[s][1], ah[s][3], al[s][1], al[s][3]);
    }
    if (c + 1 < n_chunks) load(c + 1);  // in flight during the products
    ok = ok && mbar_wait(&full[c % STAGES], c / STAGES & 1);
    if (!__syncthreads_and(ok)) break;  // (bounded wait) the same for the whole CTA
    const uint32_t w = smem_u32(smem) + c % STAGES * STAGE + lane * 16;
    constexpr int B = 4;  // expert tiles whose chains of products run side by side
#pragma unroll
    for (int n0 = 0; n0 < NTN; n0 += B) {
      if (NTN > B && (uint32_t)n0 >= nt) break;  // uniform; the last tiles of a partial group read stale bytes that go nowhere
      float acc[B][4], low[B][4];  // hi * hi, and the two small products: each is rounded by additions of its own size
#pragma unroll
      for (int n = 0; n < B; n++) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = low[n][0] = low[n][1] = low[n][2] = low[n][3] = 0.0f;
#pragma unroll
      for (uint32_t s = 0; s < STEPS; s++) {
        uint4 b[B];
#pragma unroll
        for (int n = 0; n < B; n++) b[n] = lds128(w + (n0 + n) * TILE_CHUNK + s * FRAG);
#pragma unroll
        for (int n = 0; n < B; n++) mma_acc(low[n], al[s], b[n].x, b[n].y);
#pragma unroll
        for (int n = 0; n < B; n++) mma_acc(low[n], ah[s], b[n].z, b[n].w);
#pragma unroll
        for (int n = 0; n < B; n++) mma_acc(acc[n], ah[s], b[n].x, b[n].y);
      }
#pragma unroll
      for (int n = 0; n < B; n++) {
        float(&o)[4] = sum[n0 + n];
        o[0] = fmaf(u0, acc[n][0] + low[n][0], o[0]), o[1] = fmaf(u0, acc[n][1] + low[n][1], o[1]);
        o[2] = fmaf(u1, acc[n][2] + low[n][2], o[2]), o[3] = fmaf(u1, acc[n][3] + low[n][3], o[3]);
      }
    }
    __syncthreads();  // everybody is done with the stage
    if (threadIdx.x == 0 && c + STAGES < n_chunks) issue(c + STAGES);
  }
  if (!ok) {
    if (lane == 0) atomicOr(status, MER_DEVSTAT_TIMEOUT);
    for (uint32_t s = 0; s < STAGES; s++) (void)mbar_wait(&full[s], 0), (void)mbar_wait(&full[s], 1);  // copies in flight land, or not, within a bound
  }
  float *out = logits + (size_t)blockIdx.z * T * E;
#pragma unroll
  for (int n = 0; n < NTN; n++) {
    const uint32_t e = (nt0 + n) * 8 + 2 * t;
#pragma unroll
    for (int j = 0; j < 2; j++) {
      if (e + j >= E) continue;
      const float un = __ldg(r.w_unscale + e + j);
      if (row0 < T) out[(size_t)row0 * E + e + j] = sum[n][j] * un;
      if (row1 < T) out[(size_t)row1 * E + e + j] = sum[n][2 + j] * un;
    }
  }
}

}  // namespace

// (704 x 60: weights 9.0e-8 off with the direct fp32 sums of any other width, 1.02e-7 with this)
bool router_split_supported(uint32_t D) { return D % 256 == 0; }
size_t router_split_bytes(uint32_t E, uint32_t D) { return (size_t)((E + 7) / 8 * 8) * D * 4; }

cudaError_t launch_split_router(const float *w, uint32_t E, uint32_t D, uint8_t *out, float *unscale, cudaStream_t s) {
  k_split_router<<<(E + 7) / 8 * 8, 256, 0, s>>>(w, E, D, out, unscale);
  return cudaGetLastError();
}

cudaError_t launch_router_logits(const RouterDev &r, const MoeDispatch &d, uint32_t *status, uint32_t *sets, cudaStream_t s) {
  const uint32_t E = r.num_experts, tiles = (E + 7) / 8, n_chunks = d.D / CHUNK;
  const bool wide = tiles > 8;
  const uint32_t ntn = wide ? 16 : 8;
  dim3 grid((tiles + ntn - 1) / ntn, (d.n_tokens + LG_TOKENS - 1) / LG_TOKENS);
  // slices of K until there is a CTA for every SM (the partial sets must fit the logits scratch, max_tokens x 4096 floats)
  for (uint32_t ks = 2; ks <= 16 && ks <= n_chunks; ks++)
    if (n_chunks % ks == 0 && grid.x * grid.y * ks <= 160 && (size_t)ks * E <= 4096) grid.z = ks;
  const size_t smem = (size_t)STAGES * ntn * TILE_CHUNK;
  auto kern = wide ? k_router_logits<16> : k_router_logits<8>;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  *sets = grid.z;
  kern<<<grid, LG_THREADS, smem, s>>>(r, d.x, d.n_tokens, d.D, grid.z, d.logits, status);
  return cudaGetLastError();
}
