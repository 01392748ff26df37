// Router logits of a few hundred tokens and more: logits[t][e] = x[t] . w[e], on the tensor cores at no less than fp32 precision, or in fp32 tiles
// (launch_router_logits says when).  The former:
//   * Both operands are split into f16 hi + lo parts after exact power-of-two scalings: a router row by its maximum when the router is
//     installed, a token's 64 values at a time by theirs.  Three products (hi*hi, hi*lo, lo*hi) of a chunk of 64 values are summed in the
//     tensor core, the large one in two halves, and the chunk's sum is unscaled and added in fp32: the tensor core's additions round towards zero, and a
//     whole row of 7168 values summed there would be off by 1e-5.  The parts hold
//     22 bits of values within 2^-28 of their row's (64 values') largest; a router of which a row has more than a quarter of its values below that
//     is left to fp32.
//   * The router's parts lie in mma.sync B fragment order, K permuted within every 16 values so that a lane's four are neighbours in
//     memory: a chunk of an expert tile is one bulk copy, a fragment one 128-bit load.  A fragments are made in registers from the rows of x.
//   * A CTA computes 128 tokens (16 per warp) x 8 NTN experts over a slice of K; the selection adds the slices.
// What bounds it: the legacy tensor path, 8 cycles per m16n8k16 and scheduler.
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

__device__ __forceinline__ float pow2_scale(float mx) {  // mx * scale in [2^14, 2^15); 1 for zero and non-finite rows
  if (!(mx > 0.0f) || !isfinite(mx)) return 1.0f;
  int e;
  frexpf(mx, &e);
  return ldexpf(1.0f, max(-100, min(126, 15 - e)));  // (beyond 2^115 the f16 parts overflow, and the logits become NaN)
}
// The lo part is kept 2^11 times as large: it has 11 bits of its own as long as the hi part has, down to 2^-28 of the row's largest value (unscaled: to 2^-17).  What lies
// below is off by 2^-50 of the largest.
constexpr float LO = 2048.0f;
constexpr float LEAST = 1.0f / (1 << 28);

// One router row per CTA -> its fragments, and 1 / scale.  Rows past the last expert are zeros.  `unfit` becomes nonzero for weights that the parts do not hold.
__global__ void __launch_bounds__(256) k_split_router(const float *__restrict__ w, uint32_t E, uint32_t D, uint8_t *__restrict__ out, float *__restrict__ unscale, uint32_t *unfit) {
  __shared__ float s_max[8];
  __shared__ uint32_t s_small, s_nonzero;
  const uint32_t e = blockIdx.x, n_tiles = gridDim.x / 8;
  float mx = 0.0f;
  if (threadIdx.x == 0) s_small = s_nonzero = 0;
  if (e < E)
    for (uint32_t k = threadIdx.x; k < D; k += 256) mx = nan_max(mx, fabsf(w[(size_t)e * D + k]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = nan_max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = mx;
  __syncthreads();
  for (int i = 0; i < 8; i++) mx = nan_max(mx, s_max[i]);
  const float sc = pow2_scale(mx);
  if (threadIdx.x == 0) unscale[e] = 1.0f / sc;
  uint32_t small = 0, nonzero = 0;
  for (uint32_t k = threadIdx.x; k < D; k += 256) {
    const float f = e < E ? w[(size_t)e * D + k] : 0.0f, v = f * sc;
    small += f != 0.0f && fabsf(f) < mx * LEAST, nonzero += f != 0.0f;
    const __half hi = __float2half_rn(v), lo = __float2half_rn((v - __half2float(hi)) * LO);
    const uint32_t kk = k % 16, lane = (e % 8) * 4 + kk / 4;
    __half *dst = reinterpret_cast<__half *>(out + ((size_t)(k / CHUNK) * n_tiles + e / 8) * TILE_CHUNK + k % CHUNK / 16 * FRAG + lane * 16);
    dst[kk % 4] = hi, dst[4 + kk % 4] = lo;
  }
  atomicAdd(&s_small, small), atomicAdd(&s_nonzero, nonzero);
  __syncthreads();
  if (threadIdx.x == 0 && (!(mx == 0.0f || (mx * sc >= 16384.0f && mx * sc < 32768.0f)) || s_small * 4 > s_nonzero)) *unfit = 1;
}

__device__ __forceinline__ void mma_acc(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) { mma_f16(d, a[0], a[1], a[2], a[3], b0, b1, d[0], d[1], d[2], d[3]); }
__device__ __forceinline__ float max4(float m, float4 v) { return nan_max(nan_max(nan_max(nan_max(m, fabsf(v.x)), fabsf(v.y)), fabsf(v.z)), fabsf(v.w)); }
// Four neighbouring values of a row -> its two A registers, hi and lo.
__device__ __forceinline__ void split4(float4 v, float sc, uint32_t &h0, uint32_t &h1, uint32_t &l0, uint32_t &l1) {
  v.x *= sc, v.y *= sc, v.z *= sc, v.w *= sc;  // exact
  const __half2 a = __floats2half2_rn(v.x, v.y), b = __floats2half2_rn(v.z, v.w);
  const float2 fa = __half22float2(a), fb = __half22float2(b);
  h0 = h2_bits(a), h1 = h2_bits(b);
  l0 = h2_bits(__floats2half2_rn((v.x - fa.x) * LO, (v.y - fa.y) * LO)), l1 = h2_bits(__floats2half2_rn((v.z - fb.x) * LO, (v.w - fb.y) * LO));
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
      float acc[2][B][4], low[B][4];  // hi * hi of either half, and the two small products: each is rounded by additions of its own size
#pragma unroll
      for (int n = 0; n < B; n++)
#pragma unroll
        for (int i = 0; i < 4; i++) acc[0][n][i] = acc[1][n][i] = low[n][i] = 0.0f;
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
        for (int n = 0; n < B; n++) mma_acc(acc[s * 2 / STEPS][n], ah[s], b[n].x, b[n].y);
      }
#pragma unroll
      for (int n = 0; n < B; n++)
#pragma unroll
        for (int i = 0; i < 4; i++) sum[n0 + n][i] = fmaf(i < 2 ? u0 : u1, fmaf(1.0f / LO, low[n][i], acc[0][n][i] + acc[1][n][i]), sum[n0 + n][i]);
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

// Router logits of a large batch as a tiled fp32 GEMM: logits[t][e] = x[t] . w[e].  A CTA computes TT tokens x TE experts; K
// runs in chunks of KC values that cp.async double-buffers in shared memory.  A warp owns 32 tokens x 64 experts over a
// slice of every chunk; a thread holds 8 tokens x 8 experts (rows ty + 4 i and tx + 8 j: neighbouring lanes read neighbouring
// rows, whose stride of 4 mod 32 floats keeps every 128-bit load conflict-free), i.e. 16 shared 128-bit loads per 256 FMAs.
// The slices' partial sums are added at the end in warp order.
// What bounds it is reading operand rows from L2: the 64 x 128 tile reads half as much per FMA as 32 x 64
// (4096 x 256 x 7168: 432 us with the selection).
constexpr int RL_WARPS = 8, RL_THREADS = 32 * RL_WARPS;
template <int TT, int TE, int KC>
struct LogitsTile {
  static constexpr int SPATIAL = TT / 32 * (TE / 64), SLICES = RL_WARPS / SPATIAL, SLICE_K = KC / SLICES, LD = KC + 4;
  static constexpr size_t BUF = (size_t)(TT + TE) * LD, SMEM = 2 * BUF * 4;  // floats per buffer; bytes
};
template <int TT, int TE, int KC>
__global__ void __launch_bounds__(RL_THREADS) k_router_logits_tiled(RouterDev r, MoeDispatch d, uint32_t ksplit) {
  using S = LogitsTile<TT, TE, KC>;
  constexpr int RL_TT = TT, RL_TE = TE, RL_KC = KC, RL_LD = S::LD, PIECES = KC / 4, STEP = RL_THREADS / PIECES;
  constexpr size_t RL_BUF = S::BUF;
  extern __shared__ __align__(16) float sm[];
  const uint32_t E = r.num_experts, D = d.D, T = d.n_tokens;
  const uint32_t t0 = blockIdx.y * RL_TT, e0 = blockIdx.x * RL_TE;
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t where = warp % S::SPATIAL, slice = warp / S::SPATIAL;
  const uint32_t ty = where % (TT / 32) * 32 + (lane >> 3), tx = where / (TT / 32) * 64 + (lane & 7);
  float acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int j = 0; j < 8; j++) acc[i][j] = 0.0f;
  // global -> shared: a thread copies one 16-byte piece of every STEP-th row
  const uint32_t lr = tid / PIECES, lc = tid % PIECES * 4;
  auto issue_chunk = [&](uint32_t k0, uint32_t buf) {
    float *xs = sm + buf * RL_BUF, *ws = xs + RL_TT * RL_LD;
#pragma unroll
    for (int i = 0; i < RL_TT / STEP; i++) {
      const uint32_t row = STEP * i + lr;
      const float *src = d.x + (size_t)min(t0 + row, T - 1) * D + k0 + lc;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(xs + row * RL_LD + lc)), "l"(src) : "memory");
    }
#pragma unroll
    for (int j = 0; j < RL_TE / STEP; j++) {
      const uint32_t row = STEP * j + lr;
      const float *src = r.w + (size_t)min(e0 + row, E - 1) * D + k0 + lc;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(ws + row * RL_LD + lc)), "l"(src) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // A batch of a few hundred tokens makes too few tiles for the SMs: blockIdx.z then takes one of `ksplit` slices of K
  // and writes its partial logits to set z of d.logits ([ksplit][T][E]); the selection adds the sets in order.
  const uint32_t n_chunks = D / RL_KC / ksplit, c_base = blockIdx.z * n_chunks;
  issue_chunk(c_base * RL_KC, 0);
  for (uint32_t c = 0; c < n_chunks; c++) {
    if (c + 1 < n_chunks) {
      issue_chunk((c_base + c + 1) * RL_KC, (c + 1) & 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");  // chunk c has landed (this thread's pieces)
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();  // ... and everybody else's
    const float *xs = sm + (c & 1) * RL_BUF, *ws = xs + RL_TT * RL_LD;
#pragma unroll 2
    for (int kk = 0; kk < S::SLICE_K; kk += 4) {
      const int k = slice * S::SLICE_K + kk;
      float4 a[8], b[8];
#pragma unroll
      for (int i = 0; i < 8; i++) a[i] = *reinterpret_cast<const float4 *>(xs + (ty + 4 * i) * RL_LD + k);
#pragma unroll
      for (int j = 0; j < 8; j++) b[j] = *reinterpret_cast<const float4 *>(ws + (tx + 8 * j) * RL_LD + k);
#pragma unroll
      for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 8; j++) {
          acc[i][j] = fmaf(a[i].x, b[j].x, acc[i][j]);
          acc[i][j] = fmaf(a[i].y, b[j].y, acc[i][j]);
          acc[i][j] = fmaf(a[i].z, b[j].z, acc[i][j]);
          acc[i][j] = fmaf(a[i].w, b[j].w, acc[i][j]);
        }
    }
    __syncthreads();  // the buffer may be refilled two iterations from now
  }
  // partial sums of slices 1.. through shared memory (the operand buffers are done with), added to slice 0's in order
  float *red = sm;  // [SLICES - 1][RL_TT * RL_TE]
  static_assert((S::SLICES - 1) * RL_TT * RL_TE <= 2 * RL_BUF, "the partial sums fit the operand buffers");
  if (slice > 0) {
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
      for (int j = 0; j < 8; j++) red[(slice - 1) * RL_TT * RL_TE + (ty + 4 * i) * RL_TE + tx + 8 * j] = acc[i][j];
  }
  __syncthreads();
  if (slice == 0) {
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
      for (int j = 0; j < 8; j++) {
        float v = acc[i][j];
#pragma unroll
        for (int g = 0; g < S::SLICES - 1; g++) v += red[g * RL_TT * RL_TE + (ty + 4 * i) * RL_TE + tx + 8 * j];
        const uint32_t t = t0 + ty + 4 * i, e = e0 + tx + 8 * j;
        if (t < T && e < E) d.logits[((size_t)blockIdx.z * T + t) * E + e] = v;
      }
  }
}

}  // namespace

bool router_split_supported(uint32_t D) { return D % 256 == 0; }
size_t router_split_bytes(uint32_t E, uint32_t D) { return (size_t)((E + 7) / 8 * 8) * D * 4; }

cudaError_t launch_split_router(const float *w, uint32_t E, uint32_t D, uint8_t *out, float *unscale, uint32_t *unfit, cudaStream_t s) {
  const cudaError_t e = cudaMemsetAsync(unfit, 0, 4, s);
  if (e != cudaSuccess) return e;
  k_split_router<<<(E + 7) / 8 * 8, 256, 0, s>>>(w, E, D, out, unscale, unfit);
  return cudaGetLastError();
}

cudaError_t launch_router_logits(const RouterDev &r, const MoeDispatch &d, uint32_t *status, uint32_t *sets, bool *in_parts, cudaStream_t s) {
  const uint32_t E = r.num_experts, T = d.n_tokens;
  // Slices of K until there is a CTA for every SM (the partial sets must fit the logits scratch, max_tokens x 4096 floats, and a slice is a whole number of chunks).
  auto plan = [&](uint32_t tt, uint32_t te, uint32_t kc, uint32_t most) {
    dim3 grid((E + te - 1) / te, (T + tt - 1) / tt);
    const uint32_t n_chunks = d.D / kc, tiles = grid.x * grid.y;
    for (uint32_t ks = 2; ks <= most && ks <= n_chunks; ks++)
      if (n_chunks % ks == 0 && tiles * ks <= 160 && (size_t)ks * E <= 4096) grid.z = ks;
    return grid;
  };
  // fp32 tiles: the large one where it fills the chip and the experts fill it
  using Big = LogitsTile<64, 128, 128>;
  using Small = LogitsTile<32, 64, 256>;
  const dim3 big = plan(64, 128, 128, 8), small = plan(32, 64, 256, 8);
  const bool use_big = E > 64 && (E % 128 == 0 || E > 512) && big.x * big.y * big.z >= 120;
  // Of the two the one whose error is smaller: fp32 where slices leave a thread sums of 32 terms, else the parts.  Relative error of the mixing weights against 64 bits,
  // rms, fp32 / parts, and us with the selection: 300 tokens x 128 experts of 1024 1.11e-7 / 1.20e-7, 25.6 / 33.7; of 2048 1.47e-7 / 1.62e-7, 34.6 / 36.7;
  // (64 terms) of 4096 2.43e-7 / 2.26e-7, 42.6 / 43.2; 2048 tokens x 128 of 512 1.02e-7 / 0.91e-7, 34 / 36; (256 terms) of 2048 2.95e-7 / 1.44e-7, 56 / 46;
  // 4096 x 256 of 7168 2.8e-6 / 4e-7, 432 / 211.
  const uint32_t terms = use_big ? d.D / big.z / Big::SLICES : d.D / small.z / Small::SLICES;
  *in_parts = r.w_split && terms > 32;
  if (!*in_parts) {
    const size_t smem = use_big ? Big::SMEM : Small::SMEM;
    auto kern = use_big ? k_router_logits_tiled<64, 128, 128> : k_router_logits_tiled<32, 64, 256>;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const dim3 grid = use_big ? big : small;
    *sets = grid.z;
    kern<<<grid, RL_THREADS, smem, s>>>(r, d, grid.z);
    return cudaGetLastError();
  }
  const bool wide = E > 64;
  const uint32_t ntn = wide ? 16 : 8;
  const dim3 grid = plan(LG_TOKENS, 8 * ntn, CHUNK, 16);
  const size_t smem = (size_t)STAGES * ntn * TILE_CHUNK;
  auto kern = wide ? k_router_logits<16> : k_router_logits<8>;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  *sets = grid.z;
  kern<<<grid, LG_THREADS, smem, s>>>(r, d.x, T, d.D, grid.z, d.logits, status);
  return cudaGetLastError();
}
