// One expert on the reference's flat block stream, a few tokens, no workspace beyond one row of h per token: both projections
// in ONE cooperative launch (the no-allocation entry point).  HBM-bound: an expert's bytes are read once.
//
//   * A CTA owns whole 16-row tiles (8 gate + the 8 matching up rows, then 16 down rows) and walks K in ranges of 128 (Q4_0) or
//     64 (Q8_0, short rows) blocks; partial tiles stay in shared memory between the ranges, so K needs no split over CTAs and no scratch.
//   * Two producer warps copy each tile's sixteen row pieces global -> shared with bulk async copies into rows padded so that
//     the eight rows a fragment load touches start in different banks.  A row piece that does not start on a 16-byte
//     boundary (rows that are no multiple of 256 values) is copied from the boundary below and read with a byte shift.
//   * Sixteen consumer warps split the range's blocks: every warp multiplies its few blocks of all tiles, mostly two tiles at a time, with activation
//     fragments of its own (mma B fragments, f16 hi + lo after an exact power-of-two scaling of the slice), so no warp waits
//     for another one's fragments; there the values of the next range are fetched while this one is multiplied.  Integer weights become A fragments as in kernels_stream.cu; two adjacent blocks (36 or 68
//     bytes) are loaded as aligned 32-bit words and shifted by the two bytes of the first scale.
//   * An epilogue warp adds the sixteen partial tiles of a step, and at the last range applies SiLU(gate) * up or stores the output.
//   * Every wait is bounded.  A CTA whose wait ran out latches MER_DEVSTAT_TIMEOUT and stores NaN for what it has not computed: the
//     call is asynchronous, and a caller that does not ask for the status must not take the rest for a result.
// What bounds it: the consumers' instructions, 2100 cycles a tile of 4096 values where HBM takes 1600, and 3 us each of start and grid barrier.  A
// 4096 x 14336 expert, us a call: Q4_0 and four tokens 43 / 39, Q8_0 and one token 59 / 52, with one tile at a time and fragments made from memory by
// chained shuffles (2.5 us a range, 1.4 now) / now; one warp per weight row with byte loads took 620.  Four producer warps leave the consumers 80
// registers: 43.
#include <algorithm>

#include "../../include/mer_b200.h"
#include "decode.cuh"
#include "kernels.h"
#include "ptx.cuh"

namespace {

constexpr int FC_WARPS = 16, F_PROD = 17, F_PRODS = 2,  // warp 16 is the epilogue
              F_WARPS = F_PROD + F_PRODS, F_THREADS = F_WARPS * 32;
constexpr uint32_t F_MAX_STAGES = 8, F_MAX_TILES = 16;  // tiles a CTA may own per phase
constexpr size_t F_SMEM = 226 * 1024;

template <int DT, int NT, bool ALIGNED, uint32_t RANGE_>
struct Flat {
  static constexpr uint32_t BB = DT == MER_DTYPE_Q4_0 ? MER_Q4_BLOCK_BYTES : MER_Q8_BLOCK_BYTES;
  // A warp multiplies two tiles at a time and has the values of its next range fetched ahead, with one token tile (two leave room for two stages only), but not on
  // Q4_0 rows off a 16-byte boundary: their shifted loads take the registers (8 bytes were spilled).  Us a call of four tokens, fragments from memory / both / neither: 4128 x
  // 14336 57.8 / 59.7 / 55.0, 1056 x 4128 16.7 / 18.7 / 16.7, 4000 x 14304 51.2 / 49.5 / 47.5.
  static constexpr bool BOTH = NT == 1 && (ALIGNED || DT != MER_DTYPE_Q4_0);
  static constexpr uint32_t TILES = BOTH ? 2 : 1;
  // A warp without a block of a short range makes no fragments (4128 x 14336 above 55.7 with them), except where the branch costs the loops more: Q4_0 on whole
  // 16-byte boundaries (4096 x 14336 39.3, 41.2 with the branch), and two token tiles (Q8_0, six tokens and 1792 x 3072 17.9, 18.3 with it).
  static constexpr bool SKIP = NT == 1 && (RANGE_ == 64 || !BOTH);
  static constexpr uint32_t RANGE = RANGE_, PER_WARP = RANGE / FC_WARPS;
  static constexpr uint32_t ROW = RANGE * BB + (DT == MER_DTYPE_Q4_0 ? 16 : 32);  // = 4 or 8 words mod 32
  static constexpr uint32_t STAGE = 16 * ROW;
  static constexpr uint32_t SEED_ROW = RANGE + 4;
  static constexpr uint32_t OFF_SEED = 512, OFF_RED = (OFF_SEED + 4 * NT * SEED_ROW * 4 + 127) & ~127u;
  static constexpr uint32_t OFF_ACC = OFF_RED + FC_WARPS * TILES * NT * 256, OFF_FRAG = OFF_ACC + F_MAX_TILES * NT * 256;
  static constexpr uint32_t OFF_RING = OFF_FRAG + RANGE * NT * 512;
  static constexpr uint32_t FIT = (uint32_t)((F_SMEM - 64 - OFF_RING) / STAGE), STAGES = FIT < F_MAX_STAGES ? FIT : F_MAX_STAGES;
  static constexpr uint32_t SMEM = OFF_RING + STAGES * STAGE + 64;  // a shifted load may look a few bytes past the last row
  static_assert(STAGES >= 2 * TILES, "two steps' stages at least");
};

struct FlatParams {
  const uint8_t *expert;
  const float *x;
  float *h, *out;
  uint32_t D, F, n_tokens;
  float limit;
  uint64_t wait_ns;        // limit of the wait between the projections
  uint32_t *bar, *status;  // bar[0]: arrivals, bar[1]: exits; both zero between launches
};

// B fragments of one n = 8 tile (four tokens) of PW blocks, and their seeds, from v: this lane's half of the eight values that it and the other lane of
// its token hold of a block (zeros: absent); the two swap hi and lo parts.  Returns 2^24 / scale of the token of this lane's accumulator columns.
template <int DT, int PW>
__device__ __forceinline__ float flat_fragments(float4 (&v)[PW], uint8_t *frag, uint32_t stride, float *seed) {
  const uint32_t lane = threadIdx.x & 31, t = lane & 3;
  const bool lo_lane = lane & 4;
  uint32_t most = 0;  // of the magnitudes' bits: a NaN's are above an infinity's
#pragma unroll
  for (int j = 0; j < PW; j++)
    most = max(max(max(max(most, __float_as_uint(fabsf(v[j].x))), __float_as_uint(fabsf(v[j].y))), __float_as_uint(fabsf(v[j].z))), __float_as_uint(fabsf(v[j].w)));
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) most = max(most, __shfl_xor_sync(0xffffffffu, most, o));
  // scaled to [256, 512), by 2^126 at most; non-finite activations poison the row, as they would in fp32
  const int e = min(135 - (int)(most >> 23), 126);
  const bool finite = most < 0x7f800000u;
  const float sc = most == 0 ? 1.0f : finite ? __int_as_float((e + 127) << 23) : __uint_as_float(most);
  const float un = most == 0 ? POW2_24 : finite ? POW2_24 * __int_as_float((127 - e) << 23) : POW2_24 / sc;
  float sum[PW];
#pragma unroll
  for (int j = 0; j < PW; j++) {
    v[j].x *= sc, v[j].y *= sc, v[j].z *= sc, v[j].w *= sc;  // exact (a power of two)
    sum[j] = (v[j].x + v[j].y) + (v[j].z + v[j].w);
  }
  // A block's sum over the token's eight lanes: in each step a lane hands on half of its sums, so that it ends with one block's.
  uint32_t at = 0;
#pragma unroll
  for (int o = 1, n = PW; o < 8; o <<= 1) {
    const bool upper = lane & o;
    if (n > 1) {
      n >>= 1;
#pragma unroll
      for (int j = 0; j < n; j++) {
        const float other = __shfl_xor_sync(0xffffffffu, upper ? sum[j] : sum[n + j], o);
        sum[j] = (upper ? sum[n + j] : sum[j]) + other;
      }
      at += upper ? n : 0;
    } else {
      sum[0] += __shfl_xor_sync(0xffffffffu, sum[0], o);
    }
  }
  seed[at] = -(DT == MER_DTYPE_Q4_0 ? 8.0f : 128.0f) / POW2_24 * sum[0];
#pragma unroll
  for (int j = 0; j < PW; j++) {
    float m[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
    if (DT == MER_DTYPE_Q4_0 && lo_lane) m[0] *= 0.0625f, m[1] *= 0.0625f, m[2] *= 0.0625f, m[3] *= 0.0625f;  // their nibbles sit 4 bits higher
    const __half2 h0 = __floats2half2_rn(m[0], m[2]), h1 = __floats2half2_rn(m[1], m[3]);
    const float2 f0 = __half22float2(h0), f1 = __half22float2(h1);
    const uint32_t hb0 = h2_bits(h0), hb1 = h2_bits(h1), lb0 = h2_bits(__floats2half2_rn(m[0] - f0.x, m[2] - f0.y)),
                   lb1 = h2_bits(__floats2half2_rn(m[1] - f1.x, m[3] - f1.y));
    const uint32_t g0 = __shfl_xor_sync(0xffffffffu, lo_lane ? hb0 : lb0, 4), g1 = __shfl_xor_sync(0xffffffffu, lo_lane ? hb1 : lb1, 4);
    *reinterpret_cast<uint4 *>(frag + j * stride) = lo_lane ? make_uint4(g0, g1, lb0, lb1) : make_uint4(hb0, hb1, g0, g1);
  }
  __syncwarp();  // the seeds cross lanes
  return __shfl_sync(0xffffffffu, un, t * 8);
}

// Four bytes at a byte offset that is a multiple of two.
__device__ __forceinline__ uint32_t lds_u16x2(uint32_t addr) {
  const uint32_t a = addr & ~3u;
  return __funnelshift_r(lds32(a), lds32(a + 4), (addr & 3u) * 8);
}

// ALIGNED: every row piece starts on a 16-byte boundary (d_model and d_ff multiples of 256).
template <int DT, int NT, bool ALIGNED, uint32_t RANGE>
__global__ void __launch_bounds__(F_THREADS, 1) k_flat_expert(const FlatParams p) {
  extern __shared__ __align__(128) uint8_t smem[];
  using S = Flat<DT, NT, ALIGNED, RANGE>;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g8 = lane >> 2, t = lane & 3;
  uint64_t *full = reinterpret_cast<uint64_t *>(smem), *empty = full + F_MAX_STAGES;
  uint64_t *red_full = full + 2 * F_MAX_STAGES, *red_empty = red_full + 1, *phase_ready = red_full + 2;
  volatile uint32_t *s_abort = reinterpret_cast<volatile uint32_t *>(smem + 256);
  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < S::STAGES; s++) mbar_init(&full[s], F_PRODS), mbar_init(&empty[s], FC_WARPS);
    mbar_init(red_full, FC_WARPS), mbar_init(red_empty, 1), mbar_init(phase_ready, 1);
    *s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  const size_t proj = (size_t)p.D * p.F / 32 * S::BB;
  uint32_t stage = 0, round = 0;
  bool ok = true;
  auto next_stage = [&]() {
    if (++stage == S::STAGES) stage = 0, round++;
  };
  // this CTA's tiles of a phase
  auto tiles_of = [&](int ph, uint32_t &t0, uint32_t &t1, uint32_t &kb_total) {
    const uint32_t n = ph == 0 ? p.F / 8 : p.D / 16;
    kb_total = (ph == 0 ? p.D : p.F) / 32;
    t0 = n * blockIdx.x / gridDim.x, t1 = n * (blockIdx.x + 1) / gridDim.x;
  };
  // row slot 0..15 of tile `tile` -> its first byte of block kb
  auto row_ptr = [&](int ph, uint32_t tile, uint32_t slot, uint32_t kb_total, uint32_t kb) {
    const uint32_t row = ph == 0 ? tile * 8 + (slot & 7) : tile * 16 + slot;
    return p.expert + (ph == 0 ? (slot >> 3) * proj : 2 * proj) + ((size_t)row * kb_total + kb) * S::BB;
  };

  if (warp >= F_PROD) {
    // ------------------------------------------------------------------------------------------------------ producers
    const uint32_t slot = (warp - F_PROD) * 8 + (lane & 7);
#pragma unroll 1
    for (int ph = 0; ph < 2 && ok; ph++) {
      uint32_t t0, t1, kbt;
      tiles_of(ph, t0, t1, kbt);
#pragma unroll 1
      for (uint32_t kb0 = 0; kb0 < kbt && ok; kb0 += S::RANGE) {
        const uint32_t nb = min(S::RANGE, kbt - kb0);
#pragma unroll 1
        for (uint32_t tile = t0; tile < t1; tile++) {
          if (round > 0) ok = mbar_wait(&empty[stage], (round - 1) & 1, s_abort);
          if (*s_abort) ok = false;
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          const uint8_t *src = row_ptr(ph, tile, slot, kbt, kb0);
          const uint32_t shift = ALIGNED ? 0u : (uint32_t)((size_t)src & 15u), bytes = ALIGNED ? nb * S::BB : (shift + nb * S::BB + 15u) & ~15u;
          uint32_t total = lane < 8 ? bytes : 0u;
          if (!ALIGNED) {
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
          } else {
            total = 8 * bytes;
          }
          if (lane == 0) mbar_expect_tx(&full[stage], total);
          __syncwarp();
          if (lane < 8) bulk_g2s(smem + S::OFF_RING + stage * S::STAGE + slot * S::ROW, src - shift, bytes, &full[stage]);
          next_stage();
        }
      }
    }
    if (!ok) {
      if (lane == 0) *s_abort = 1;
      // copies in flight get a bounded chance to land before the CTA's memory is released: the last phase of every stage
      // issued to (which stays open, to the limit, only if the other producer stopped before it)
      for (uint32_t s = 0; s < S::STAGES; s++)
        if (s < stage || round > 0) mbar_drain(&full[s], (s < stage ? round : round - 1) & 1, 10000000ull);
    }
  } else if (warp < FC_WARPS) {
    // ------------------------------------------------------------------------------------------------------ consumers
    uint8_t *s_frag = smem + S::OFF_FRAG + warp * (S::PER_WARP * NT * 512) + lane * 16;
    float *s_seed = reinterpret_cast<float *>(smem + S::OFF_SEED) + warp * S::PER_WARP;
    const uint32_t frags = smem_u32(s_frag), seeds = smem_u32(s_seed) + t * (S::SEED_ROW * 4);
    float2 *s_red = reinterpret_cast<float2 *>(smem + S::OFF_RED) + warp * (S::TILES * NT * 32) + lane;
    const uint32_t lane_value = (DT == MER_DTYPE_Q4_0 ? 4 : 8) * t + ((lane & 4) ? (DT == MER_DTYPE_Q4_0 ? 16 : 4) : 0);
    uint32_t n_red = 0;
#pragma unroll 1
    for (int ph = 0; ph < 2 && ok; ph++) {
      uint32_t t0, t1, kbt;
      tiles_of(ph, t0, t1, kbt);
      if (ph == 1) {
        ok = mbar_wait(phase_ready, 0);  // every CTA's rows of h are visible
        if (*s_abort) ok = false;
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
      }
      const float *act = ph == 0 ? p.x : p.h;
      if (t0 == t1) continue;
      // this warp's blocks of a range, whole pairs
      auto share = [&](uint32_t kb0, uint32_t &b0) {
        const uint32_t nb = min(S::RANGE, kbt - kb0), width = ((nb + FC_WARPS - 1) / FC_WARPS + 1) & ~1u;
        b0 = warp * width;
        return nb > b0 ? min(width, nb - b0) : 0u;
      };
      float4 v[S::PER_WARP];  // this lane's values of a range
      auto fetch = [&](uint32_t kb0, int n) {
        uint32_t b0;
        const uint32_t mine = share(kb0, b0), tok = n * 4 + (g8 >> 1);
        const float *row = act + (size_t)tok * kbt * 32 + (kb0 + b0) * 32 + lane_value;
#pragma unroll
        for (uint32_t j = 0; j < S::PER_WARP; j++)
          v[j] = tok < p.n_tokens && j < mine ? *reinterpret_cast<const float4 *>(row + j * 32) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      };
      if (S::BOTH) fetch(0, 0);
#pragma unroll 1
      for (uint32_t kb0 = 0; kb0 < kbt && ok; kb0 += S::RANGE) {
        uint32_t b0;
        const uint32_t mine = share(kb0, b0);
        float un[NT];
#pragma unroll
        for (int n = 0; n < NT; n++) {
          if (!S::BOTH) fetch(kb0, n);
          un[n] = 0.0f;
          if (!S::SKIP || mine > 0) un[n] = flat_fragments<DT>(v, s_frag + n * 512, NT * 512, s_seed + (n * 4 + (g8 >> 1)) * S::SEED_ROW);
        }
        if (S::BOTH && kb0 + S::RANGE < kbt) fetch(kb0 + S::RANGE, 0);  // the next range's values arrive while this one is multiplied
#pragma unroll 1
        for (uint32_t tile = t0; tile < t1; tile += S::TILES) {
          const uint32_t live = min(S::TILES, t1 - tile);
          float acc[S::TILES][NT][4];
          // row addresses of slots g8 and g8 + 8 (and where their first block starts inside the copied piece)
          uint32_t r0[S::TILES], r1[S::TILES];
#pragma unroll
          for (uint32_t u = 0; u < S::TILES; u++) {
#pragma unroll
            for (int n = 0; n < NT; n++) acc[u][n][0] = acc[u][n][1] = acc[u][n][2] = acc[u][n][3] = 0.0f;
            if (u > 0 && u >= live) break;
            r0[u] = smem_u32(smem) + S::OFF_RING + stage * S::STAGE + g8 * S::ROW, r1[u] = r0[u] + 8 * S::ROW;
            if (!ALIGNED) {
              r0[u] += (uint32_t)((size_t)row_ptr(ph, tile + u, g8, kbt, kb0) & 15u);
              r1[u] += (uint32_t)((size_t)row_ptr(ph, tile + u, g8 + 8, kbt, kb0) & 15u);
            }
            r0[u] += b0 * S::BB, r1[u] += b0 * S::BB;
            if (ok) ok = mbar_wait(&full[stage], round & 1);
            next_stage();
          }
          ok = __all_sync(0xffffffffu, ok);
          if (ok) {
#pragma unroll 1
            for (uint32_t j = 0; j < mine; j += 2) {
              uint4 b[NT][2];
              float sd[NT][2];
#pragma unroll
              for (int n = 0; n < NT; n++)
#pragma unroll
                for (int i = 0; i < 2; i++) {
                  b[n][i] = lds128(frags + ((j + i) * NT + n) * 512);
                  sd[n][i] = __uint_as_float(lds32(seeds + n * (4 * S::SEED_ROW * 4) + (j + i) * 4));
                }
#pragma unroll
              for (uint32_t u = 0; u < S::TILES; u++) {
                if (u > 0 && u >= live) break;
                uint32_t a[2][2][4];  // [block][row slot g8, g8 + 8]
                uint32_t s[2][2];     // f16 scale bits
#pragma unroll
                for (int r = 0; r < 2; r++) {
                  const uint32_t rp = r ? r1[u] : r0[u];
                  if (DT == MER_DTYPE_Q4_0) {
                    uint32_t q0, q1;
                    if (ALIGNED) {
                      const uint32_t w0 = lds32(rp + 4 * t), w1 = lds32(rp + 4 * t + 4);
                      q0 = __funnelshift_r(w0, w1, 16), q1 = lds32(rp + 20 + 4 * t);
                      s[0][r] = lds32(rp) & 0xffffu, s[1][r] = lds32(rp + 16) >> 16;
                    } else {
                      q0 = lds_u16x2(rp + 2 + 4 * t), q1 = lds_u16x2(rp + 20 + 4 * t);
                      s[0][r] = lds_u16x2(rp) & 0xffffu, s[1][r] = lds_u16x2(rp + 16) >> 16;
                    }
                    unpack_q4(q0, a[0][r]), unpack_q4(q1, a[1][r]);
                  } else {
                    uint32_t l0, h0, l1, h1;
                    if (ALIGNED) {
                      const uint32_t w0 = lds32(rp + 8 * t), w1 = lds32(rp + 8 * t + 4), w2 = lds32(rp + 8 * t + 8);
                      l0 = __funnelshift_r(w0, w1, 16), h0 = __funnelshift_r(w1, w2, 16);
                      l1 = lds32(rp + 36 + 8 * t), h1 = lds32(rp + 40 + 8 * t);
                      s[0][r] = lds32(rp) & 0xffffu, s[1][r] = lds32(rp + 32) >> 16;
                    } else {
                      l0 = lds_u16x2(rp + 2 + 8 * t), h0 = lds_u16x2(rp + 6 + 8 * t), l1 = lds_u16x2(rp + 36 + 8 * t), h1 = lds_u16x2(rp + 40 + 8 * t);
                      s[0][r] = lds_u16x2(rp) & 0xffffu, s[1][r] = lds_u16x2(rp + 32) >> 16;
                    }
                    unpack_q8(l0, h0, a[0][r]), unpack_q8(l1, h1, a[1][r]);
                  }
                }
                if (j + 1 >= mine) s[1][0] = s[1][1] = 0;  // no second block: stale bytes against zero fragments
#pragma unroll
                for (int n = 0; n < NT; n++) {
                  float c1[2][4], c2[2][4];
#pragma unroll
                  for (int i = 0; i < 2; i++)
                    mma_f16(c1[i], a[i][0][0], a[i][1][0], a[i][0][1], a[i][1][1], b[n][i].x, b[n][i].y, sd[n][i], 0.0f, sd[n][i], 0.0f);
#pragma unroll
                  for (int i = 0; i < 2; i++)
                    mma_f16(c2[i], a[i][0][2], a[i][1][2], a[i][0][3], a[i][1][3], b[n][i].z, b[n][i].w, c1[i][0], c1[i][1], c1[i][2], c1[i][3]);
#pragma unroll
                  for (int i = 0; i < 2; i++) {
                    const float d0 = __half2float(__ushort_as_half((unsigned short)s[i][0])), d1 = __half2float(__ushort_as_half((unsigned short)s[i][1]));
                    acc[u][n][0] = fmaf(d0, c2[i][0], acc[u][n][0]);
                    acc[u][n][1] = fmaf(d0, c2[i][1], acc[u][n][1]);
                    acc[u][n][2] = fmaf(d1, c2[i][2], acc[u][n][2]);
                    acc[u][n][3] = fmaf(d1, c2[i][3], acc[u][n][3]);
                  }
                }
                r0[u] += 2 * S::BB, r1[u] += 2 * S::BB;
              }
            }
          }
          __syncwarp();
          if (lane < live) mbar_arrive(&empty[stage >= live - lane ? stage - (live - lane) : stage + S::STAGES - (live - lane)]);
          if (ok && n_red > 0) ok = mbar_wait(red_empty, (n_red - 1) & 1);
          ok = __all_sync(0xffffffffu, ok);
          n_red++;
#pragma unroll
          for (uint32_t u = 0; u < S::TILES; u++)
#pragma unroll
            for (int n = 0; n < NT; n++)
              s_red[(u * NT + n) * 32] = make_float2((acc[u][n][0] + acc[u][n][1]) * un[n], (acc[u][n][2] + acc[u][n][3]) * un[n]);
          __syncwarp();
          if (lane == 0) mbar_arrive(red_full);
        }
      }
    }
    if (!ok && lane == 0) *s_abort = 1;
  } else {
    // ------------------------------------------------------------------------------------------------------- epilogue
    const float2 *s_red = reinterpret_cast<const float2 *>(smem + S::OFF_RED) + lane;
    float2 *s_acc = reinterpret_cast<float2 *>(smem + S::OFF_ACC) + lane;
    const bool clamp = p.limit > 0.0f && isfinite(p.limit);
    uint32_t n_red = 0;
#pragma unroll 1
    for (int ph = 0; ph < 2; ph++) {
      uint32_t t0, t1, kbt;
      tiles_of(ph, t0, t1, kbt);
#pragma unroll 1
      for (uint32_t kb0 = 0; kb0 < kbt && ok; kb0 += S::RANGE) {
        const bool first = kb0 == 0, last = kb0 + S::RANGE >= kbt;
#pragma unroll 1
        for (uint32_t first_tile = t0; first_tile < t1 && ok; first_tile += S::TILES) {
          ok = mbar_wait(red_full, n_red++ & 1) && !*s_abort;
          ok = __all_sync(0xffffffffu, ok);
#pragma unroll
          for (uint32_t un = 0; un < S::TILES * NT; un++) {
            const uint32_t u = un / NT, n = un % NT, tile = first_tile + u;
            if (tile >= t1) break;
            float2 o = make_float2(0.0f, 0.0f);
#pragma unroll
            for (int s = 0; s < FC_WARPS; s++) {
              const float2 v = s_red[((s * S::TILES + u) * NT + n) * 32];
              o.x += v.x, o.y += v.y;
            }
            float2 &a = s_acc[((tile - t0) * NT + n) * 32];
            if (!first) o.x += a.x, o.y += a.y;
            const uint32_t tok = n * 4 + t;
            if (!last) {
              a = o;
            } else if (tok < p.n_tokens) {
              if (ph == 0) {  // row slots 0..7 are gate rows, 8..15 the matching up rows
                float gate = o.x;
                if (clamp && gate == gate) gate = fminf(fmaxf(gate, -p.limit), p.limit);
                p.h[(size_t)tok * p.F + tile * 8 + g8] = __fdividef(gate, 1.0f + __expf(-gate)) * o.y;
              } else {
                p.out[(size_t)tok * p.D + tile * 16 + g8] = o.x;
                p.out[(size_t)tok * p.D + tile * 16 + 8 + g8] = o.y;
              }
            }
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(red_empty);
        }
      }
      __syncwarp();
      if (!ok) {  // fail closed: NaN rows of h make every output NaN
        const float nan = __uint_as_float(0x7fc00000u);
        const uint32_t rows = ph == 0 ? 8 : 16, len = ph == 0 ? p.F : p.D;
        float *dst = ph == 0 ? p.h : p.out;
        for (uint32_t i = lane; i < (t1 - t0) * rows * p.n_tokens; i += 32)
          dst[(size_t)(i / ((t1 - t0) * rows)) * len + t0 * rows + i % ((t1 - t0) * rows)] = nan;
        __syncwarp();
      }
      if (ph == 0) {  // h is exchanged between all CTAs
        if (lane == 0) {
          __threadfence();
          atomicAdd(p.bar, 1u);
          const uint64_t since = global_ns();
          while (*(volatile uint32_t *)p.bar < gridDim.x && ok)
            if (global_ns() - since > p.wait_ns) ok = false;
          __threadfence();
        }
        ok = __all_sync(0xffffffffu, ok);
        if (lane == 0) {
          if (!ok) *s_abort = 1;
          mbar_arrive(phase_ready);
        }
      }
    }
    if (!ok && lane == 0) *s_abort = 1;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (*s_abort) atomicOr(p.status, MER_DEVSTAT_TIMEOUT);
    // the last CTA to leave re-arms the barrier (everybody has passed it)
    __threadfence();
    if (atomicInc(p.bar + 1, gridDim.x - 1) == gridDim.x - 1) p.bar[0] = 0;
  }
}

template <int DT, int NT, bool ALIGNED, uint32_t RANGE>
cudaError_t launch_flat(FlatParams p, int sm_count, cudaStream_t s) {
  using S = Flat<DT, NT, ALIGNED, RANGE>;
  if ((p.F / 8 + sm_count - 1) / sm_count > F_MAX_TILES || (p.D / 16 + sm_count - 1) / sm_count > F_MAX_TILES) return cudaErrorNotSupported;
  auto kern = k_flat_expert<DT, NT, ALIGNED, RANGE>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM);
  if (e != cudaSuccess) return e;
  void *args[] = {&p};
  return cudaLaunchCooperativeKernel((const void *)kern, dim3(sm_count), dim3(F_THREADS), args, S::SMEM, s);
}
template <int DT>
cudaError_t launch_flat_dt(const FlatParams &p, int sm_count, cudaStream_t s) {
  const bool aligned = p.D % 256 == 0 && p.F % 256 == 0;
  constexpr uint32_t RANGE = DT == MER_DTYPE_Q4_0 ? 128 : 64;
  if (p.n_tokens > 4) return aligned ? launch_flat<DT, 2, true, RANGE>(p, sm_count, s) : launch_flat<DT, 2, false, RANGE>(p, sm_count, s);
  if (!aligned) return launch_flat<DT, 1, false, RANGE>(p, sm_count, s);
  // One range of at most 64 blocks: half the values a warp holds for 128, and no more tiles than CTAs to speak of.  Us a call of one token, ranges of 128 / 64:
  // 2048 x 768 12.6 / 10.6 (10.6 with fragments from memory), 1024 x 1024 11.6 / 10.6, 2048 x 1536 12.6 / 11.6, 2048 x 2048 12.6 both.
  return std::max(p.D, p.F) <= 2048 ? launch_flat<DT, 1, true, 64>(p, sm_count, s) : launch_flat<DT, 1, true, RANGE>(p, sm_count, s);
}

}  // namespace

bool flat_expert_supported(const void *expert, const void *x, uint32_t D, uint32_t F, uint32_t n_tokens) {
  // whole blocks per row: row pieces then never reach past the blob's last 16-byte line
  return D % 32 == 0 && F % 32 == 0 && n_tokens <= 8 && ((size_t)expert & 15u) == 0 && ((size_t)x & 15u) == 0;
}

cudaError_t launch_flat_expert(int dtype, const uint8_t *expert, const float *x, float *h, float *out, uint32_t D, uint32_t F, uint32_t n_tokens, float limit,
                               uint64_t wait_ns, uint32_t *bar, uint32_t *status, int sm_count, cudaStream_t s) {
  const FlatParams p{expert, x, h, out, D, F, n_tokens, limit, wait_ns, bar, status};
  return dtype == MER_DTYPE_Q4_0 ? launch_flat_dt<MER_DTYPE_Q4_0>(p, sm_count, s) : launch_flat_dt<MER_DTYPE_Q8_0>(p, sm_count, s);
}
