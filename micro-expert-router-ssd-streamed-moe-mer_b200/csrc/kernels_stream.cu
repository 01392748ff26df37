// Streaming expert FFN for decode-sized token groups (a few tokens per expert).
//
// One cooperative launch runs a layer's gate/up phase, the hidden values, the down phase and the weighted combine:
//   * Experts are resident in the tile-major fragment layout of layout.cuh (the reference's blocks, permuted at admission).  A stage
//     of the ring is one chunk of each of an item's sixteen 16-row tiles, each chunk moved global -> shared memory by ONE bulk async
//     copy (cp.async.bulk, completion on an mbarrier): every byte of an expert is read from HBM once, as a linear stream.  The
//     copies run on into the down phase while the grid finishes the gate/up phase.
//   * Warps unpack the integer part of the weights straight into f16 mma.sync A fragments.  A 4-bit or 8-bit field masked into the
//     low mantissa bits of an f16 IS the subnormal value q * 2^-24 (q * 2^-20 for a field at bits 4..7), so unpacking is one ALU
//     instruction per two weights and the integers are exact.  The zero point (8 for Q4_0, 128 for the biased Q8_0 byte) is added
//     four blocks at a time as the product of the blocks' scales and -zp * sum(x_block).
//   * Activations come as images (act_image.cuh): f16 hi + lo parts (22 significant bits) after an exact power-of-two scaling of
//     the row; hi and lo are two columns of the n=8 MMA tile, so one tile carries 4 tokens.  Products are exact, accumulation is
//     fp32 in the tensor core.  A CTA copies those of the unit, i.e. (pass, K split), that comes next while it multiplies the present
//     one; warps meet at no barrier when units change.
//   * The per-block f16 scale d is applied in fp32 when a block's partial is folded into the row accumulator: acc += d * partial
//     (the ordering of matmul_q4_0.wgsl:65-85 in the reference).
//
// Work is cut into items (token pass, K split, group of 16 tiles), which a scheduler warp claims for its CTA; each of the eight
// consumer warps owns two tiles of the item over its K range, so no warp ever waits for another one's partial sums.  Load balance
// comes from splitting K across CTAs and from taking over items: partial sums go to scratch and are added behind grid-wide barriers
// (SiLU(gate) * up between the phases, the weighted combine at the end; kernels of their own where a cooperative launch is
// refused), always in the same order, so results are deterministic; no atomics on data.  Every wait is bounded: on expiry the warp
// stops computing, the CTA latches MER_DEVSTAT_TIMEOUT, drains its copies in flight and returns.
//
// What bounds it: instructions of the consumers, next to HBM.  On sm_100 an m16n8k16 holds a scheduler's FMA pipe for 8 cycles, and an ALU
// operation half a warp-instruction slot: a block of 16 rows costs 2.25 MMAs, 4 FMAs and 10 (Q4_0) or 8 (Q8_0) ALU operations at up to
// four tokens.  With the copies left out the gate/up phase of 64 tokens on 128 experts of 2048 x 768 took 74 us of 79, with the
// products left out 65; 16 tokens on 8 of 4096 x 14336 122 of 128, and 91.  Q8_0 bytes with the sign bit to flip (12 ALU operations
// a block) took 10 % more of the whole layer, and one tile a warp in sixteen warps 6 % more on 16 tokens of 256 x 7168 x 2048
// (even elsewhere).  Around the loops: barriers 1.3 us each, hidden values 2 to 3, combine 3 to 5, first activations 3 to 4.  FFN of a layer, two launches
// before and one now: 64 tokens on 128 experts of 2048 x 768 146 -> 129 us, 16 on 256 of 7168 x 2048 500 -> 470, one on 128 of
// 2048 x 768 (with its routing) 37 -> 28.
#include "kernels.h"

#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

#include "../../include/mer_b200.h"
#include "act_image.cuh"
#include "decode.cuh"
#include "layout.cuh"
#include "ptx.cuh"
#include "route.cuh"

namespace {

constexpr int ITEM_TILES = 16, WARP_TILES = 2, CONSUMER_WARPS = ITEM_TILES / WARP_TILES, CONSUMERS = CONSUMER_WARPS * 32;
constexpr int PRODUCER_WARPS = 2;  // each issues the bulk copies of half a stage's tiles: one warp alone was busy ~90 % of the time
constexpr int SCHED_WARP = CONSUMER_WARPS + PRODUCER_WARPS;  // claims the CTA's items and fetches their activations
constexpr int THREADS = (SCHED_WARP + 1) * 32;
constexpr uint32_t QUEUE = 3;
constexpr uint32_t HEADER_BYTES = 1024;  // of `Header`
constexpr uint32_t N_BARRIERS = 4;       // grid-wide barriers of a launch, one counter each

constexpr int TAIL_NONE = 0, TAIL_COMBINE = 1, TAIL_REDUCE = 2;

struct PhaseParams {
  uint32_t packed_tiles;  // 16-row tiles of the projection (F / 8 for gate/up, D / 16 for down)
  uint32_t kb_total;      // 32-weight blocks per row
  uint32_t kb_split;      // blocks per K split (kb_total when n_ksplit == 1)
  uint32_t n_ksplit;
};

struct StreamParams {
  MoeDispatch d;
  PhaseParams ph[2];         // gate/up, down
  uint32_t phases;           // bit mask of the phases this launch runs
  uint32_t kc;               // blocks per pipeline stage
  uint32_t n_stages;
  uint32_t chunk_stride;     // bytes between the 16-row tile chunks of a stage (kc * 16 * block bytes)
  uint32_t n_frag;           // activation buffers (1 or 2)
  uint32_t queue[2];         // items a CTA claims ahead in either phase (1 .. QUEUE)
  uint32_t frag_cols;        // fragment arrays of a buffer: 2 * min(4 * NT, most tokens of any group)
  uint32_t frag_bytes;       // bytes of a buffer
  float *parts;              // gate/up partials [n_ksplit][P][2][F]
  float *down_parts;         // with K split, down partials [n_ksplit][P x D]: the same place, except with LOCAL
  int sync;                  // cooperative launch: the grid-wide steps below run here (0: kernels of their own follow)
  int tail;                  // after the down phase, by the whole grid after a grid-wide barrier:
                             // TAIL_COMBINE: out[token] = weighted sum of its pairs' outputs in slot order;
                             // TAIL_REDUCE (K split): y[pair] = sum of its partials, grouped pairs only
  uint32_t *bar;             // [N_BARRIERS] arrival counters
};

// Words between two columns of zero-point terms: 4 mod 8, so that the eight columns and four blocks a warp reads together lie in
// different banks.
__host__ __device__ constexpr uint32_t seed_words(uint32_t kb_split) { return ((kb_split + 7) & ~7u) + 4; }
// Bytes between the fragment arrays of two columns: 64 mod 128, which keeps the 128-bit loads of a warp free of conflicts.
__host__ __device__ constexpr uint32_t frag_stride(uint32_t kb_split) { return (kb_split * 64 & ~127u) + 64 + (kb_split & 1) * 128; }

__device__ __forceinline__ void consumer_sync() { asm volatile("bar.sync 1, %0;" ::"n"(CONSUMERS) : "memory"); }
// Ordinary stores before bulk copies that read them, and the other way round.
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async;" ::: "memory"); }

template <int DT>
struct BlockBytes {
  static constexpr uint32_t value = DT == MER_DTYPE_Q4_0 ? MER_Q4_BLOCK_BYTES : MER_Q8_BLOCK_BYTES;
};

// Grid-wide barrier among the consumers of a cooperative launch.  The increments of one use add up to 2^31: the counter's top bit
// flips when the last CTA arrives, and nothing has to clear it.  For that every CTA arrives at each of its launch's barriers
// exactly once, whatever happened before.  Waits are bounded by wall-clock time.
__device__ bool grid_barrier(uint32_t *counter, uint32_t *s_ok, uint32_t *status) {
  consumer_sync();  // this CTA's stores are issued
  if (threadIdx.x == 0) {
    const uint32_t old = arrive_acq_rel(counter, blockIdx.x == 0 ? 0x80000000u - (gridDim.x - 1) : 1u);
    const uint64_t t0 = global_ns();
    bool ok = false;
    for (uint32_t polls = 0; !ok; polls++) {
      ok = ((load_acquire(counter) ^ old) & 0x80000000u) != 0;
      if (!ok && (polls & 31) == 31 && global_ns() - t0 > 2000000000ull) break;
    }
    if (!ok) atomicOr(status, MER_DEVSTAT_TIMEOUT);
    *s_ok = ok;
  }
  consumer_sync();
  return *(volatile uint32_t *)s_ok != 0;
}

// Four hidden values of a pair from each of `R` places: h = SiLU(sum of gate partials) * (sum of up partials), partials added in K-split order.  Place r
// is f0 + r * step; zeros from f_end on.
template <int R>
__device__ __forceinline__ void hidden_values(const MoeDispatch &d, const float *parts, uint32_t n_ksplit, uint32_t pair, uint32_t f0, uint32_t step, uint32_t f_end, float4 (&h)[R]) {
  const uint32_t F = d.F;
  const float *base = parts + (size_t)pair * 2 * F + f0;
  const size_t part = (size_t)d.n_tokens * d.slots * 2 * F;
  float4 up[R];
#pragma unroll
  for (int r = 0; r < R; r++) h[r] = up[r] = make_float4(0, 0, 0, 0);
#pragma unroll (8 / R)
  for (uint32_t k = 0; k < n_ksplit; k++, base += part) {  // loads of several splits in flight, added in order
#pragma unroll
    for (int r = 0; r < R; r++) {
      if (f0 + r * step >= f_end) continue;
      const float4 a = __ldcg(reinterpret_cast<const float4 *>(base + r * step)), b = __ldcg(reinterpret_cast<const float4 *>(base + F + r * step));
      h[r].x += a.x, h[r].y += a.y, h[r].z += a.z, h[r].w += a.w;
      up[r].x += b.x, up[r].y += b.y, up[r].z += b.z, up[r].w += b.w;
    }
  }
  const bool clamp = d.swiglu_limit > 0.0f && isfinite(d.swiglu_limit);
  auto one = [&](float gate, float u) {
    if (clamp && gate == gate) gate = fminf(fmaxf(gate, -d.swiglu_limit), d.swiglu_limit);
    return __fdividef(gate, 1.0f + __expf(-gate)) * u;
  };
#pragma unroll
  for (int r = 0; r < R; r++) h[r] = make_float4(one(h[r].x, up[r].x), one(h[r].y, up[r].y), one(h[r].z, up[r].z), one(h[r].w, up[r].w));
}
// Largest magnitude of a warp's values, as float bits: a NaN sorts above all numbers.
__device__ __forceinline__ uint32_t abs_bits(float v) { return __float_as_uint(v) & 0x7fffffffu; }
__device__ __forceinline__ uint32_t max_bits(uint32_t m, float4 v) { return max(max(max(max(m, abs_bits(v.x)), abs_bits(v.y)), abs_bits(v.z)), abs_bits(v.w)); }
// Power of two that brings a largest magnitude into [2^14, 2^15): f16 hi + lo parts then have 22 bits for all values within 2^-16 of it (2^-12 in
// the upper nibbles' places of Q4_0), and an error of 2^-39 (2^-35) of it below.  It has to be that of the values themselves: a bound made of
// max |gate| and max |up| is too large by e^20 where an expert's gates lie near -20.
__device__ __forceinline__ float hidden_scale(uint32_t bits) {
  const float mx = __uint_as_float(bits);
  if (mx == 0.0f) return 1.0f;
  if (!isfinite(mx)) return __int_as_float(0x7fc00000);  // non-finite values poison the row, as they would in fp32
  int e;
  frexpf(mx, &e);
  return ldexpf(1.0f, min(127, 15 - e));
}
// The step between the phases: the hidden values into the activation images of the down phase.  A unit is what one down item multiplies, the values of a pair in
// one K split, with a scale of its own: `chunks` runs of 128 values, by a team of so many of the CTA's warps that each has HIDDEN_RUNS of them in
// registers, or of more while no warp has to take a second unit.  A team of eight keeps the rest of longer units in `stash` (kb_split x 128 bytes).
// What bounds it is the round trip of a unit's loads.  Us a layer, with a scale per row from a bound, 128 values a unit, / this: 64 tokens on 128 experts of
// 2048 x 768 154 / 153; 43 on 96 of 1792 x 6656 378 / 368; 16 on 8 of 4096 x 14336 216 / 213; one on those (eight units of 3584 values) 67.0 / 67.4.
// Four runs in registers spill: the first 155.
constexpr int HIDDEN_RUNS = 2;
__device__ __forceinline__ void hidden_units(const MoeDispatch &d, const float *parts, uint32_t n_ksplit, const PhaseParams &down, uint32_t cta, uint32_t n_ctas, uint32_t warp,
                                             uint32_t lane, uint32_t *s_red, float4 *stash) {
  const bool some = d.expected_pairs != 0;  // under expert parallelism a fraction of all pairs is here
  const uint32_t chunks = (down.kb_split + 3) / 4, units = (some ? __ldcg(d.offsets + d.n_groups) : d.n_tokens * d.slots) * down.n_ksplit;
  uint32_t W = 1, log_w = 0;
  while (W < CONSUMER_WARPS && W < chunks && (W * HIDDEN_RUNS < chunks || units * W < n_ctas * (CONSUMER_WARPS / 2))) W *= 2, log_w++;
  const uint32_t teams = CONSUMER_WARPS >> log_w, team = warp >> log_w, member = warp & (W - 1), span = W * HIDDEN_RUNS * 32;
  uint32_t *red = s_red + team * W;
#pragma unroll 1
  for (uint32_t u = cta * teams + team, odd = 0; u < units; u += n_ctas * teams, odd ^= CONSUMER_WARPS) {
    const uint32_t i = u / down.n_ksplit, ks = u % down.n_ksplit, pair = some ? __ldcg(d.perm + i) : i, kb0 = ks * down.kb_split, n4 = min(down.kb_split, down.kb_total - kb0) * 8;
    const uint32_t turns = (n4 + span - 1) / span;
    float4 h[HIDDEN_RUNS];
    uint32_t m = 0;
#pragma unroll 1
    for (uint32_t turn = 0; turn < turns; turn++) {
      hidden_values<HIDDEN_RUNS>(d, parts, n_ksplit, pair, (kb0 * 8 + turn * span + member * 32 + lane) * 4, W * 128, (kb0 * 8 + n4) * 4, h);
#pragma unroll
      for (int r = 0; r < HIDDEN_RUNS; r++) {
        m = max_bits(m, h[r]);
        if (turn + 1 < turns) stash[turn * span + (r * W + member) * 32 + lane] = h[r];
      }
    }
    m = __reduce_max_sync(0xffffffffu, m);
    if (W > 1) {  // (two sets of words in turn: one barrier a unit)
      if (lane == 0) red[odd + member] = m;
      asm volatile("bar.sync %0, %1;" ::"r"(2 + team), "r"(W * 32) : "memory");
      m = __reduce_max_sync(0xffffffffu, lane < W ? red[odd + lane] : 0u);
    }
    const float sc = hidden_scale(m);
    if (member == 0 && lane == 0) d.h_un[pair * down.n_ksplit + ks] = POW2_24 / sc;
    const ImageRow row(d.h, d.act_seeds, pair, d.F);
#pragma unroll 1
    for (uint32_t turn = turns; turn-- > 0;) {  // the last one's values are still there
#pragma unroll
      for (int r = 0; r < HIDDEN_RUNS; r++) {
        const uint32_t q = turn * span + (r * W + member) * 32 + lane;
        if (turn + 1 < turns) h[r] = stash[q];
        const float4 v = make_float4(h[r].x * sc, h[r].y * sc, h[r].z * sc, h[r].w * sc);
        image_store4(d.dtype, v, kb0 * 8 + q, q < n4, row.hi, row.lo, row.seed_hi, row.seed_lo);
      }
    }
  }
}

// After all CTAs have left their outputs of the down phase: the arithmetic of k_combine / k_reduce_ksplit, spread over the consumers of the grid.
__device__ void ffn_stream_tail(const StreamParams &p) {
  const MoeDispatch &d = p.d;
  const uint32_t P = d.n_tokens * d.slots, n_ksplit = p.ph[1].n_ksplit;
  if (p.tail == TAIL_COMBINE) {
    const uint32_t D4 = d.D / 4;
    const float4 *yp = reinterpret_cast<const float4 *>(n_ksplit > 1 ? p.down_parts : d.y);
    const size_t part4 = (size_t)P * D4;
#pragma unroll 1
    for (uint32_t e = blockIdx.x * CONSUMERS + threadIdx.x; e < d.n_tokens * D4; e += gridDim.x * CONSUMERS) {
      const uint32_t token = e / D4, i4 = e % D4;
      float4 acc = make_float4(0, 0, 0, 0);
      auto add_residual = [&]() {  // hidden + routed sum, before the shared expert's slot (model.rs:2742-2763)
        const float4 r = __ldg(reinterpret_cast<const float4 *>(d.residual) + (size_t)token * D4 + i4);
        acc.x = __fadd_rn(r.x, acc.x), acc.y = __fadd_rn(r.y, acc.y), acc.z = __fadd_rn(r.z, acc.z), acc.w = __fadd_rn(r.w, acc.w);
      };
      // four slots at a time: their loads are in flight together (one by one, the eight partial sums of two slots took 3 us)
      constexpr uint32_t S = 4;
#pragma unroll 1
      for (uint32_t s0 = 0; s0 < d.slots; s0 += S) {
        float w[S];
        float4 yv[S];
        // (an unfilled slot's output is whatever the scratch holds and is not added)
        uint32_t who[S];
#pragma unroll
        for (uint32_t j = 0; j < S; j++) {
          const size_t pr = (size_t)token * d.slots + min(s0 + j, d.slots - 1);
          w[j] = d.pair_weight[pr], who[j] = d.pair_expert[pr];
          yv[j] = __ldcg(yp + pr * D4 + i4);
        }
#pragma unroll 1
        for (uint32_t k = 1; k < n_ksplit; k++) {
#pragma unroll
          for (uint32_t j = 0; j < S; j++) {
            const float4 t = __ldcg(yp + (size_t)k * part4 + ((size_t)token * d.slots + min(s0 + j, d.slots - 1)) * D4 + i4);
            yv[j].x += t.x, yv[j].y += t.y, yv[j].z += t.z, yv[j].w += t.w;
          }
        }
#pragma unroll
        for (uint32_t j = 0; j < S; j++)
          if (s0 + j >= d.slots || who[j] == MER_NONE) w[j] = 0.0f;
#pragma unroll
        for (uint32_t j = 0; j < S; j++) {
          if (d.residual && s0 + j == d.routed_slots && s0 + j < d.slots) add_residual();
          if (w[j] == 0.0f) continue;
          acc.x = __fadd_rn(acc.x, __fmul_rn(w[j], yv[j].x));
          acc.y = __fadd_rn(acc.y, __fmul_rn(w[j], yv[j].y));
          acc.z = __fadd_rn(acc.z, __fmul_rn(w[j], yv[j].z));
          acc.w = __fadd_rn(acc.w, __fmul_rn(w[j], yv[j].w));
        }
      }
      if (d.residual && d.routed_slots >= d.slots) add_residual();
      reinterpret_cast<float4 *>(d.out)[(size_t)token * D4 + i4] = acc;
    }
  } else if (p.tail == TAIL_REDUCE) {
    // per-pair outputs of the pairs that ran here (under expert parallelism: a fraction of all pairs)
    const uint32_t D4 = d.D / 4, n_here = d.offsets[d.n_groups];
    const float4 *yp = reinterpret_cast<const float4 *>(p.down_parts);
    const size_t part4 = (size_t)P * D4;
#pragma unroll 1
    for (uint32_t e = blockIdx.x * CONSUMERS + threadIdx.x; e < n_here * D4; e += gridDim.x * CONSUMERS) {
      const size_t pr = d.perm[e / D4];
      const uint32_t i4 = e % D4;
      float4 yv = __ldcg(yp + pr * D4 + i4);
#pragma unroll 1
      for (uint32_t k = 1; k < n_ksplit; k++) {
        const float4 t = __ldcg(yp + (size_t)k * part4 + pr * D4 + i4);
        yv.x += t.x, yv.y += t.y, yv.z += t.z, yv.w += t.w;
      }
      reinterpret_cast<float4 *>(d.y)[pr * D4 + i4] = yv;
    }
  }
}

// --------------------------------------------------------------------------- main kernel
// An item as the scheduler hands it to the CTA's other warps.
struct __align__(16) Item {
  uint32_t tile, ks;    // group of 16 tiles, K split
  uint32_t unit;        // running number of its (pass, K split) in this CTA: whose activations it wants
  uint32_t more;        // 0: there are no more items in this phase
  const uint8_t *base;  // the expert's payload, null = not resident
};

// The start of shared memory.
struct Header {
  uint64_t full[8], empty[8];             // [n_stages] the ring's stages
  uint64_t frag_full[2], frag_empty[2];   // [n_frag] the activation buffers
  uint64_t hidden;                        // the hidden rows are there
  uint64_t built;                         // LOCAL: the item's hidden values are in shared memory
  uint64_t q_full[QUEUE], q_empty[QUEUE]; // the item queue
  uint32_t abort, ok;
  uint32_t other_status;                  // ROUTE: where CTAs but the first leave the router's status bits
  uint32_t info[2];                       // tokens of the unit's pass
  uint32_t pair[2 * 8];                   // pair index of each of them
  float un[2 * 8];                        // its 2^24 / scale
  uint32_t red[2 * CONSUMER_WARPS];       // the warps' maxima in the making of hidden values
  Item item[QUEUE];
  const uint8_t *base[32];                // ROUTE: payload of every pass,
  uint32_t slot[32];                      //   its slot
};
static_assert(sizeof(Header) <= HEADER_BYTES, "");

// Claims items for a CTA.  The grouping kernel cut the phase's items, ordered (pass, K split, tile), into one contiguous range per CTA,
// balanced by the tokens of the passes.  A CTA takes its own from the front and, when they are used up, those of the CTA that has most
// left from the back: SMs reach HBM at different speeds, and the slowest of them finished 10 to 17 us behind the others
// (of 80 to 130, a phase of 16 to 64 tokens).  Who runs an item changes no result.  Whole warp.
struct Claims {
  const uint32_t *bounds;
  uint64_t *taken;  // low half: from the front, high half: from the back; the first item of a range is its owner's
  uint32_t beg, n_own, n_items, per, more, lane;  // per, more: without a table of bounds, the first `more` CTAs have per + 1 items, the others per
  bool first = true, own = true;
  __device__ Claims(const StreamParams &p, int phase, uint32_t n_passes, uint32_t lane_) : lane(lane_) {
    const PhaseParams &f = p.ph[phase];
    n_items = n_passes * f.n_ksplit * ((f.packed_tiles + ITEM_TILES - 1) / ITEM_TILES);
    bounds = p.d.route_here ? nullptr : p.d.item_bounds + phase * MER_MAX_CTAS1, taken = p.d.taken + phase * MER_MAX_CTAS1;
    per = n_items / gridDim.x, more = n_items - per * gridDim.x;
    beg = bound(blockIdx.x), n_own = bound(blockIdx.x + 1) - beg;
  }
  __device__ uint32_t bound(uint32_t cta) const { return bounds ? min(n_items, bounds[cta]) : per * cta + min(cta, more); }
  // Next item, or MER_NONE.
  __device__ uint32_t next() {
    if (own) {
      if (first) {
        first = false;
        if (n_own) return beg;
      }
      uint64_t old = 0;
      if (lane == 0 && n_own > 1) old = atomicAdd(reinterpret_cast<unsigned long long *>(taken + blockIdx.x), 1ull);
      const uint32_t front = __shfl_sync(0xffffffffu, (uint32_t)old, 0), back = __shfl_sync(0xffffffffu, (uint32_t)(old >> 32), 0);
      if (n_own > 1 && front + back < n_own - 1) return beg + 1 + front;
      own = false;
    }
    for (;;) {  // ends: every failed attempt means that somebody else took an item
      uint32_t best = 0, from = 0, end = 0;
#pragma unroll 1
      for (uint32_t c = lane; c < gridDim.x; c += 32) {
        const uint64_t v = *(volatile uint64_t *)(taken + c);
        const uint32_t b = bound(c), e = bound(c + 1), gone = (uint32_t)v + (uint32_t)(v >> 32) + 1;
        if (e - b > gone && e - b - gone > best) best = e - b - gone, from = c, end = e;
      }
      const uint32_t most = __reduce_max_sync(0xffffffffu, best);
      if (most == 0) return MER_NONE;
      const uint32_t who = __ffs(__ballot_sync(0xffffffffu, best == most)) - 1;
      uint32_t item = MER_NONE;
      if (lane == who) {
        const uint64_t old = atomicAdd(reinterpret_cast<unsigned long long *>(taken + from), 1ull << 32);
        const uint32_t n = end - bound(from);
        if ((uint32_t)old + (uint32_t)(old >> 32) + 1 < n) item = end - 1 - (uint32_t)(old >> 32);
      }
      item = __shfl_sync(0xffffffffu, item, who);
      if (item != MER_NONE) return item;
    }
  }
};

// Routing of a dispatch of one token by the scheduler of every CTA, from the router kernel's logits: passes of one pair each, in slot order.  All
// CTAs come to the same selection; the first one writes it down.  What it saves is the router's last CTA: arrivals, its tables' way through L2 and a
// round trip for them.  `scratch`: 2 x 256 floats, `word`: where the other CTAs' status bits go.  Returns the number of passes.
__device__ __forceinline__ uint32_t route_token_here(const MoeDispatch &d, float *scratch, const uint8_t **s_base, uint32_t *s_slot, uint32_t *word, uint32_t lane) {
  const RouterDev &r = d.route;
  for (uint32_t i = lane; i < r.num_experts; i += 32) scratch[i] = __ldcg(d.logits + i);
  __syncwarp();
  uint32_t *status = blockIdx.x == 0 ? d.status : word;
  const Pick pick = r.num_experts <= 128 ? route_token_reg<4>(r, scratch, scratch + 256, status) : route_token_reg<8>(r, scratch, scratch + 256, status);
  const bool routed = lane < r.top_k;
  const uint32_t eid = routed ? (pick.id == MER_NONE ? MER_NONE : r.id_base + pick.id) : lane < d.slots ? r.shared_expert_id : MER_NONE;
  const uint32_t valid = __ballot_sync(0xffffffffu, eid != MER_NONE), pass = __popc(valid & ((1u << lane) - 1)), n = __popc(valid);
  if (eid != MER_NONE) s_base[pass] = eid < d.max_experts ? d.expert_ptr[eid] : nullptr, s_slot[pass] = lane;
  if (blockIdx.x == 0) {
    if (lane < d.slots) d.pair_expert[lane] = eid, d.pair_weight[lane] = routed ? pick.weight : r.shared_scale ? *r.shared_scale : 1.0f;
    if (eid != MER_NONE) d.perm[pass] = lane;
    if (lane == 0) d.offsets[d.n_groups] = d.n_passes[0] = n;
  }
  __syncwarp();
  fence_async();  // the scratch is a stage of the ring
  return n;
}

// RAGGED: the last group of 16 tiles is not full, or K or a stage is no multiple of four blocks (the checks cost the even shapes 1 to 3 %).
// ROUTE: the scheduler selects the experts of the only token.  LOCAL: at most one down item a CTA, which makes the hidden values that the item wants in
// its own shared memory: no hidden rows in memory, no second barrier between the phases, no copy.  (Parameters and not branches: the code of either
// beside the loops cost 16 tokens on 8 experts of 4096 x 14336 4 %.)
template <int DT, int NT, bool RAGGED, bool ROUTE, bool LOCAL>
__device__ __forceinline__ void ffn_stream_body(const StreamParams &p) {
  extern __shared__ __align__(128) uint8_t smem[];
  constexpr uint32_t BB = BlockBytes<DT>::value;
  const MoeDispatch &d = p.d;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  Header &hd = *reinterpret_cast<Header *>(smem);
  uint64_t *const full = hd.full, *const empty = hd.empty, *const frag_full = hd.frag_full, *const frag_empty = hd.frag_empty;
  uint64_t *const hidden = &hd.hidden, *const built = &hd.built, *const q_full = hd.q_full, *const q_empty = hd.q_empty;
  uint32_t *const s_abort = &hd.abort, *const s_ok = &hd.ok, *const s_info = hd.info, *const s_pair = hd.pair, *const s_red = hd.red;
  float *const s_un = hd.un;
  Item *const s_item = hd.item;
  const uint8_t **const s_base = hd.base;
  uint32_t *const s_slot = hd.slot;
  uint8_t *s_frag = smem + HEADER_BYTES;                        // [n_frag] x {fragments [frag_cols][frag_stride], zero-point terms [frag_cols][seed_words]}
  uint8_t *s_stage = s_frag + (size_t)p.n_frag * p.frag_bytes;  // [n_stages][16 tiles][chunk_stride]
  const uint32_t stage_bytes = ITEM_TILES * p.chunk_stride;

  if (threadIdx.x < 2) s_info[threadIdx.x] = 0;
  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < p.n_stages; s++) {
      mbar_init(&full[s], PRODUCER_WARPS);
      mbar_init(&empty[s], CONSUMER_WARPS);
    }
    for (uint32_t s = 0; s < 2; s++) mbar_init(&frag_full[s], 2), mbar_init(&frag_empty[s], CONSUMER_WARPS);
    for (uint32_t s = 0; s < QUEUE; s++) mbar_init(&q_full[s], 1), mbar_init(&q_empty[s], CONSUMER_WARPS + PRODUCER_WARPS);
    mbar_init(hidden, 1), mbar_init(built, CONSUMER_WARPS);
    *s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  grid_dep_wait();
  grid_dep_launch();
  __syncthreads();

  // The CTA's next item as every warp but the scheduler's sees it; a slot is free again when all have read it.
  uint32_t q_slot = 0, q_round = 0;
  auto next_item = [&](Item &it, uint32_t depth) -> bool {
    bool ok = __all_sync(0xffffffffu, mbar_wait(&q_full[q_slot], q_round & 1));
    if (ok) it = s_item[q_slot];
    __syncwarp();
    if (lane == 0) mbar_arrive(&q_empty[q_slot]);
    if (++q_slot >= depth) q_slot = 0, q_round++;
    return ok;
  };

  const size_t proj_bytes = (size_t)d.D * d.F / 32 * BB;

  if (warp >= CONSUMER_WARPS && warp < SCHED_WARP) {
    // ------------------------------ weight producers: warp h, lane m < 8 copies the chunk of tile 8h + m of every stage.  They run on
    // into the down phase while the consumers still wait for its activations.
    constexpr uint32_t TILES_PER_PRODUCER = ITEM_TILES / PRODUCER_WARPS;
    const uint32_t my_tile = (warp - CONSUMER_WARPS) * TILES_PER_PRODUCER + (lane % TILES_PER_PRODUCER);
    uint32_t stage = 0, round = 0;
    bool ok = true;
#pragma unroll 1
    for (int phase = 0; phase < 2; phase++) {
      if (!(p.phases >> phase & 1)) continue;
      const size_t tile_bytes = (size_t)p.ph[phase].kb_total * 16 * BB;  // one packed 16-row tile, all of K
      const uint32_t packed_tiles = p.ph[phase].packed_tiles;
      const uint32_t kb_split = p.ph[phase].kb_split, kb_total = p.ph[phase].kb_total;
#pragma unroll 1
      while (ok) {
        Item it;
        ok = next_item(it, QUEUE);
        if (!ok || !it.more) break;
        if (!it.base) continue;  // consumers skip the same item
        const uint32_t kb0 = it.ks * kb_split, kbn = min(kb_split, kb_total - kb0);
        // item -> packed tiles 16*tile .. 16*tile + 15 of the phase's region
        const uint8_t *src = it.base + (phase == 0 ? 0 : 2 * proj_bytes) + (size_t)(ITEM_TILES * it.tile + my_tile) * tile_bytes;
        // tiles of this producer that exist (none: the stage's other half still completes the barrier's second arrival)
        const uint32_t first = ITEM_TILES * it.tile + (warp - CONSUMER_WARPS) * TILES_PER_PRODUCER;
        const uint32_t live = !RAGGED ? TILES_PER_PRODUCER : first >= packed_tiles ? 0u : min(TILES_PER_PRODUCER, packed_tiles - first);
        for (uint32_t c0 = 0; c0 < kbn && ok; c0 += p.kc) {
          const uint32_t nb = min(p.kc, kbn - c0);
          if (round > 0) ok = mbar_wait(&empty[stage], (round - 1) & 1);
          if (*(volatile uint32_t *)s_abort) ok = false;
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          if (lane == 0) mbar_expect_tx(&full[stage], live * nb * 16 * BB);
          __syncwarp();
          if (lane < live)
            bulk_g2s(s_stage + (size_t)stage * stage_bytes + my_tile * p.chunk_stride, src + (size_t)(kb0 + c0) * 16 * BB, nb * 16 * BB,
                     &full[stage]);
          if (++stage == p.n_stages) stage = 0, round++;
        }
      }
    }
    if (!ok) {
      if (lane == 0) {
        *(volatile uint32_t *)s_abort = 1;
        atomicOr(d.status, MER_DEVSTAT_TIMEOUT);
      }
      // drain: give copies already in flight a bounded chance to land before the CTA's memory is released
      for (uint32_t s = 0; s < p.n_stages; s++) (void)mbar_wait(&full[s], 0), (void)mbar_wait(&full[s], 1);
    }
    return;
  }

  if (warp == SCHED_WARP) {
    // ------------------------------ scheduler: claims items, and for each new unit, i.e. (pass, K split), fetches the activations: lane l
    // copies part l % 4 (hi fragments, lo fragments, their zero-point terms) of the pass's token l / 4.
    const uint32_t n_passes = ROUTE ? route_token_here(d, reinterpret_cast<float *>(s_stage), s_base, s_slot, &hd.other_status, lane) : *d.n_passes;
    uint32_t unit = 0, slot = 0, round = 0;
    bool ok = true;
    const uint32_t tok = lane >> 2, part = lane & 3;
    fence_async();
#pragma unroll 1
    for (int phase = 0; phase < 2; phase++) {
      if (!(p.phases >> phase & 1)) continue;
      const PhaseParams &f = p.ph[phase];
      const uint32_t n_tiles = (f.packed_tiles + ITEM_TILES - 1) / ITEM_TILES, K = phase == 0 ? d.D : d.F;
      const uint32_t stride = frag_stride(f.kb_split), words = seed_words(f.kb_split), ahead = p.queue[phase];
      Claims claims(p, phase, n_passes, lane);
      uint32_t cur_pp = MER_NONE, cur_ks = MER_NONE, pair = 0, count = 0;
      const uint8_t *base = nullptr, *src = nullptr;
      bool wait_hidden = phase == 1 && (p.phases & 1);  // the hidden rows come from all CTAs of this launch
#pragma unroll 1
      while (ok) {
        // no more than `ahead` items beyond the one that the slowest warp has begun
        const uint32_t entry = round * QUEUE + slot;
        if (entry >= ahead) ok = mbar_wait(&q_empty[(entry - ahead) % QUEUE], ((entry - ahead) / QUEUE) & 1);
        if (*(volatile uint32_t *)s_abort) ok = false;
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        const uint32_t item = claims.next();
        const bool more = item != MER_NONE;
        const uint32_t tile = item % n_tiles, ks = (item / n_tiles) % f.n_ksplit, pp = item / n_tiles / f.n_ksplit;
        const bool new_unit = more && (pp != cur_pp || ks != cur_ks);
        if (new_unit && pp != cur_pp) {
          if (ROUTE) {
            base = s_base[pp], count = 1, pair = s_slot[pp];
          } else {
            const PassDesc &pass = d.pass_desc[pp];
            base = pass.base, count = pass.count;
            pair = pass.pair[tok];
          }
          if (tok < count) {
            const ImageRow row(phase == 0 ? d.x_rows : d.h, d.act_seeds, phase == 0 ? pair / d.slots : pair, K);
            src = part == 0 ? row.hi : part == 1 ? row.lo : reinterpret_cast<const uint8_t *>(part == 2 ? row.seed_hi : row.seed_lo);
          }
        }
        // the weight producers may start on it while its activations are fetched
        if (lane == 0) {
          s_item[slot] = Item{tile, ks, unit + (new_unit ? 1u : 0u), more ? 1u : 0u, base};
          mbar_arrive(&q_full[slot]);
        }
        __syncwarp();
        if (++slot == QUEUE) slot = 0, round++;
        if (!more) break;
        if (!new_unit) continue;
        cur_pp = pp, cur_ks = ks;
        const uint32_t buf = p.n_frag == 2 ? unit & 1 : 0, use = p.n_frag == 2 ? unit >> 1 : unit;
        unit++;
        if (wait_hidden) {
          ok = mbar_wait(hidden, 0);
          fence_async();
          wait_hidden = false;
        }
        if (ok && use > 0) ok = mbar_wait(&frag_empty[buf], (use - 1) & 1);
        if (*(volatile uint32_t *)s_abort) ok = false;
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        const uint32_t kb0 = ks * f.kb_split, kbn = min(f.kb_split, f.kb_total - kb0), seed_bytes = ((kbn + 3) & ~3u) * 4;
        const bool copies = !(LOCAL && phase == 1);
        if (lane == 0) mbar_expect_tx(&frag_full[buf], copies ? count * 2 * (kbn * 64 + seed_bytes) : 0);
        __syncwarp();
        if (tok < count && !copies) {
          if (part == 0) s_pair[buf * 8 + tok] = pair;
        } else if (tok < count) {
          uint8_t *dst = s_frag + buf * p.frag_bytes;
          const uint32_t col = 2 * tok + (part & 1);
          if (part < 2)
            bulk_g2s(dst + col * stride, src + (size_t)kb0 * 64, kbn * 64, &frag_full[buf]);
          else
            bulk_g2s(dst + p.frag_cols * stride + col * words * 4, src + (size_t)kb0 * 4, seed_bytes, &frag_full[buf]);
          if (part == 0) s_pair[buf * 8 + tok] = pair, s_un[buf * 8 + tok] = __ldcg(phase == 0 ? d.x_un + pair / d.slots : d.h_un + pair * f.n_ksplit + ks);
        }
        if (lane == 0) s_info[buf] = count;
        __syncwarp();
        if (lane == 0) mbar_arrive(&frag_full[buf]);
      }
    }
    if (!ok) {
      if (lane == 0) {
        *(volatile uint32_t *)s_abort = 1;
        atomicOr(d.status, MER_DEVSTAT_TIMEOUT);
      }
      for (uint32_t s = 0; s < p.n_frag; s++) (void)mbar_wait(&frag_full[s], 0), (void)mbar_wait(&frag_full[s], 1);
    }
    return;
  }

  // ---------------------------------------------------------------------- consumer warps
  const uint32_t g = lane >> 2, t = lane & 3;
  const uint32_t piece16 = packed_piece(g, t) * 16;  // byte offset of this lane's 16-byte piece inside a block record
  const uint32_t stage0 = smem_u32(s_stage) + warp * WARP_TILES * p.chunk_stride;  // this warp's first tile chunk in stage 0
  // scales {row slot g, slot g+8} of block t of four, from the record of the first
  const uint32_t scale4 = DT == MER_DTYPE_Q4_0 ? (t >> 1) * 576 + 512 + g * 8 + (t & 1) * 4 : t * 544 + 512 + g * 4;
  const size_t n_pairs = (size_t)d.n_tokens * d.slots;
  uint32_t stage = 0, round = 0, builds = 0;
  bool ready = false;  // the stage has been seen full
  // A warp whose bounded wait expired goes "dead": it takes no more items, and no part in the grid-wide steps but their barriers,
  // which so always see all consumer warps.
  bool dead = false;

#pragma unroll 1
  for (int phase = 0; phase < 2; phase++) {
  if (!(p.phases >> phase & 1)) continue;
  const uint32_t packed_tiles = p.ph[phase].packed_tiles, stride = frag_stride(p.ph[phase].kb_split), words = seed_words(p.ph[phase].kb_split);
  const bool k_is_split = p.ph[phase].n_ksplit > 1;
  const uint32_t kb_split = p.ph[phase].kb_split, kb_total = p.ph[phase].kb_total;
  uint32_t cur_unit = 0, pcount = 1, buf = 0;  // units count from 1
  uint32_t fa[NT], ia[NT];  // where column g / token t of each N-tile lives
  auto leave_unit = [&]() {
    __syncwarp();
    if (lane == 0) mbar_arrive(&frag_empty[buf]);
  };
#pragma unroll 1
  while (!dead) {
    Item it;
    if (!next_item(it, QUEUE)) {
      dead = true;
      break;
    }
    if (!it.more) break;
    const uint32_t tile = it.tile, kbn = min(kb_split, kb_total - it.ks * kb_split);

    if (it.unit != cur_unit) {
      if (cur_unit) leave_unit();  // done with the previous unit's activations
      cur_unit = it.unit;
      const uint32_t u = cur_unit - 1, use = p.n_frag == 2 ? u >> 1 : u;
      buf = p.n_frag == 2 ? u & 1 : 0;
      dead = !__all_sync(0xffffffffu, mbar_wait(&frag_full[buf], use & 1));
      if (dead) break;
      pcount = *(volatile uint32_t *)&s_info[buf];
      if (LOCAL && phase == 1) {
        uint8_t *frag = s_frag + buf * p.frag_bytes;
        float *seeds = reinterpret_cast<float *>(frag + p.frag_cols * stride);
        // a run of 128 values a warp at most (one_down_item)
        const uint32_t chunks = (kbn + 3) / 4, tok = warp / chunks, q = warp % chunks * 32 + lane;
        const bool mine = tok < pcount, inside = mine && q < kbn * 8;
        auto meet = [&]() {
          __syncwarp();
          if (lane == 0) mbar_arrive(built);
          dead = dead || !__all_sync(0xffffffffu, mbar_wait(built, builds++ & 1));
        };
        const uint32_t f0 = it.ks * kb_split * 32;
        float4 h[1];
        hidden_values<1>(d, p.parts, p.ph[0].n_ksplit, s_pair[buf * 8 + (mine ? tok : 0)], f0 + q * 4, 0, mine ? f0 + kbn * 32 : 0, h);
        float4 &v = h[0];
        const uint32_t most = __reduce_max_sync(0xffffffffu, max_bits(0, v));
        if (lane == 0) s_red[warp] = most;
        meet();
        if (mine) {
          const float sc = hidden_scale(__reduce_max_sync(0xffffffffu, lane < chunks ? s_red[tok * chunks + lane] : 0u));
          v.x *= sc, v.y *= sc, v.z *= sc, v.w *= sc;
          image_store4(DT, v, q, inside, frag + 2 * tok * stride, frag + (2 * tok + 1) * stride, seeds + 2 * tok * words, seeds + (2 * tok + 1) * words);
          if (q == 0) s_un[buf * 8 + tok] = POW2_24 / sc;
        }
        meet();
        if (dead) break;
      }
      // an MMA output column depends on its own B column only, and the columns of absent tokens are never written out: they
      // read the last one that exists
      const uint32_t frag0 = smem_u32(s_frag) + buf * p.frag_bytes, seed0 = frag0 + p.frag_cols * stride;
#pragma unroll
      for (int n = 0; n < NT; n++) {
        const uint32_t col = min(n * 8 + g, 2 * pcount - 1);
        fa[n] = frag0 + t * 16 + col * stride;
        ia[n] = seed0 + t * 4 + col * words * 4;
      }
    }
    if (!it.base) {
      if (threadIdx.x == 0) atomicOr(d.status, MER_DEVSTAT_RESIDENCY_MISS);
      // fail closed: zero outputs for this item
      const uint32_t rows_per_tile = phase == 0 ? 8u : 16u, rows_here = rows_per_tile * ITEM_TILES;
      for (uint32_t i = threadIdx.x; i < rows_here * pcount; i += CONSUMERS) {
        const uint32_t pair = s_pair[buf * 8 + i / rows_here], row = tile * rows_here + i % rows_here;
        if (RAGGED && row >= packed_tiles * rows_per_tile) continue;
        if (phase == 0) {
          float *gp = p.parts + ((size_t)it.ks * n_pairs + pair) * 2 * d.F;
          gp[row] = 0.0f, gp[d.F + row] = 0.0f;
        } else {
          (k_is_split ? p.down_parts : d.y)[((size_t)it.ks * n_pairs + pair) * d.D + row] = 0.0f;
        }
      }
      continue;
    }

    float acc[WARP_TILES][NT][4];
#pragma unroll
    for (int j = 0; j < WARP_TILES; j++)
#pragma unroll
      for (int n = 0; n < NT; n++) acc[j][n][0] = acc[j][n][1] = acc[j][n][2] = acc[j][n][3] = 0.0f;
    const uint32_t n_live = (pcount + 3) >> 2;  // N-tiles that hold tokens

    // The zero point's share of `left` (at most 4) blocks: acc += scales[16 rows x 4 blocks] * terms[4 blocks x 8 columns] in
    // one MMA (a scale's 11 bits are exact in tf32, a term is two columns, hi and lo).  As the initial value of every
    // block's own MMA it cost four register moves a block, a sixth of the loop's instructions.
    auto do_zero = [&](uint32_t rec, uint32_t kb, uint32_t left, bool single_last, auto nl) {
      constexpr int NL = decltype(nl)::value;  // N-tiles that hold tokens, 0: n_live
      const bool in = !RAGGED || t < left;
      uint32_t sa = rec + scale4;
      if (RAGGED && DT == MER_DTYPE_Q4_0 && single_last && t + 1 == left) sa = rec + (t >> 1) * 576 + 256 + g * 4;  // odd K: half a pair record
      uint32_t term[NT];
#pragma unroll
      for (int n = 0; n < NT; n++) term[n] = in && (NL ? n < NL : n == 0 || (uint32_t)n < n_live) ? lds32(ia[n] + kb * 4) : 0u;
#pragma unroll
      for (int j = 0; j < WARP_TILES; j++) {
        const float2 sc = h2_to_f2(in ? lds32(sa + j * p.chunk_stride) : 0u);
#pragma unroll
        for (int n = 0; n < NT; n++) {
          if (NL ? n >= NL : (n > 0 && (uint32_t)n >= n_live)) break;  // uniform
          mma_tf32(acc[j][n], __float_as_uint(sc.x), __float_as_uint(sc.y), term[n]);
        }
      }
    };

    // two adjacent blocks (kb, kb + 1; kb even) of both row slots of the warp's tiles against every live N-tile.
    // rec = shared address of the pair's first record in the first tile's chunk.
    auto do_pair = [&](uint32_t rec, uint32_t kb, auto nl) {
      constexpr int NL = decltype(nl)::value;
      uint4 bf0[NT], bf1[NT];
#pragma unroll
      for (int n = 0; n < NT; n++) {
        if (NL ? n >= NL : (n > 0 && (uint32_t)n >= n_live)) break;  // uniform
        bf0[n] = lds128(fa[n] + kb * 64), bf1[n] = lds128(fa[n] + kb * 64 + 64);
      }
#pragma unroll
      for (int j = 0; j < WARP_TILES; j++) {
        const uint32_t r = rec + j * p.chunk_stride;
        uint32_t a0[4], a0h[4], a1[4], a1h[4];  // block kb: slots g / g+8; block kb+1: slots g / g+8
        float2 d0, d1;                          // {scale slot g, scale slot g+8} of each block
        if (DT == MER_DTYPE_Q4_0) {
          const uint4 w = lds128(r + piece16);
          const uint2 sc = lds64(r + 512 + g * 8);
          unpack_q4(w.x, a0), unpack_q4(w.y, a0h), unpack_q4(w.z, a1), unpack_q4(w.w, a1h);
          d0 = h2_to_f2(sc.x), d1 = h2_to_f2(sc.y);
        } else {
          const uint4 w0 = lds128(r + piece16), w1 = lds128(r + 544 + piece16);
          const uint32_t sc0 = lds32(r + 512 + g * 4), sc1 = lds32(r + 544 + 512 + g * 4);
          unpack_q8_biased(w0.x, w0.y, a0), unpack_q8_biased(w0.z, w0.w, a0h), unpack_q8_biased(w1.x, w1.y, a1), unpack_q8_biased(w1.z, w1.w, a1h);
          d0 = h2_to_f2(sc0), d1 = h2_to_f2(sc1);
        }
#pragma unroll
        for (int n = 0; n < NT; n++) {
          if (NL ? n >= NL : (n > 0 && (uint32_t)n >= n_live)) break;  // uniform
          float c1[4], c2[4], e1[4], e2[4];
          mma_f16(c1, a0[0], a0h[0], a0[1], a0h[1], bf0[n].x, bf0[n].y, 0.0f, 0.0f, 0.0f, 0.0f);
          mma_f16(e1, a1[0], a1h[0], a1[1], a1h[1], bf1[n].x, bf1[n].y, 0.0f, 0.0f, 0.0f, 0.0f);
          mma_f16(c2, a0[2], a0h[2], a0[3], a0h[3], bf0[n].z, bf0[n].w, c1[0], c1[1], c1[2], c1[3]);
          mma_f16(e2, a1[2], a1h[2], a1[3], a1h[3], bf1[n].z, bf1[n].w, e1[0], e1[1], e1[2], e1[3]);
          float(&o)[4] = acc[j][n];
          o[0] = fmaf(d0.x, c2[0], o[0]), o[1] = fmaf(d0.x, c2[1], o[1]), o[2] = fmaf(d0.y, c2[2], o[2]), o[3] = fmaf(d0.y, c2[3], o[3]);
          o[0] = fmaf(d1.x, e2[0], o[0]), o[1] = fmaf(d1.x, e2[1], o[1]), o[2] = fmaf(d1.y, e2[2], o[2]), o[3] = fmaf(d1.y, e2[3], o[3]);
        }
      }
    };

    // the last block of an odd K, alone: a single record (Q4_0: half a pair record)
    auto do_last = [&](uint32_t rec, uint32_t kb) {
#pragma unroll 1
      for (int j = 0; j < WARP_TILES; j++) {
        const uint32_t r = rec + j * p.chunk_stride;
        uint32_t a[4], ah[4];
        float2 ds;
        if (DT == MER_DTYPE_Q4_0) {
          const uint2 w = lds64(r + (piece16 >> 1));
          ds = h2_to_f2(lds32(r + 256 + g * 4));
          unpack_q4(w.x, a), unpack_q4(w.y, ah);
        } else {
          const uint4 w = lds128(r + piece16);
          ds = h2_to_f2(lds32(r + 512 + g * 4));
          unpack_q8_biased(w.x, w.y, a), unpack_q8_biased(w.z, w.w, ah);
        }
#pragma unroll
        for (int n = 0; n < NT; n++) {
          if (n > 0 && (uint32_t)n >= n_live) break;  // uniform
          const uint4 bf = lds128(fa[n] + kb * 64);
          float c1[4], c2[4];
          mma_f16(c1, a[0], ah[0], a[1], ah[1], bf.x, bf.y, 0.0f, 0.0f, 0.0f, 0.0f);
          mma_f16(c2, a[2], ah[2], a[3], ah[3], bf.z, bf.w, c1[0], c1[1], c1[2], c1[3]);
#pragma unroll
          for (int k = 0; k < WARP_TILES; k++)
            if (k == j) {
              float(&o)[4] = acc[k][n];
              o[0] = fmaf(ds.x, c2[0], o[0]), o[1] = fmaf(ds.x, c2[1], o[1]), o[2] = fmaf(ds.y, c2[2], o[2]), o[3] = fmaf(ds.y, c2[3], o[3]);
            }
        }
      }
    };

    // (a tile past the projection's last computes on stale bytes; it is not written)
    const bool my_tile_exists = !RAGGED || ITEM_TILES * tile + WARP_TILES * warp < packed_tiles;
    for (uint32_t c0 = 0; c0 < kbn; c0 += p.kc) {
      const uint32_t nb = min(p.kc, kbn - c0);
      if (!ready) dead = !__all_sync(0xffffffffu, mbar_wait(&full[stage], round & 1));
      if (dead) break;
      // the look at the next stage's barrier takes 100 to 200 cycles, which pass while this one is multiplied
      const uint32_t next = stage + 1 == p.n_stages ? 0 : stage + 1;
      ready = mbar_test(&full[next], (next == 0 ? round + 1 : round) & 1);
      if (my_tile_exists) {
        constexpr uint32_t PAIR_BYTES = 2 * 16 * BB;  // 576 (Q4_0) / 1088 (Q8_0)
        uint32_t rec = stage0 + stage * stage_bytes;
        using Live = std::integral_constant<int, 0>;
        using One = std::integral_constant<int, 1>;
        using All = std::integral_constant<int, NT>;
        // Four blocks per iteration keep independent MMA chains in flight, in loops of their own for one N-tile and for two.
        if (!RAGGED && (NT == 1 || n_live == 1)) {
#pragma unroll 1
          for (uint32_t b = 0; b < nb; b += 4, rec += 2 * PAIR_BYTES) {
            do_zero(rec, c0 + b, 4, false, One{});
            do_pair(rec, c0 + b, One{});
            do_pair(rec + PAIR_BYTES, c0 + b + 2, One{});
          }
        } else if (!RAGGED) {
#pragma unroll 1
          for (uint32_t b = 0; b < nb; b += 4, rec += 2 * PAIR_BYTES) {
            do_zero(rec, c0 + b, 4, false, All{});
            do_pair(rec, c0 + b, All{});
            do_pair(rec + PAIR_BYTES, c0 + b + 2, All{});
          }
        } else
#pragma unroll 1
        for (uint32_t b = 0; b < nb; b += 4, rec += 2 * PAIR_BYTES) {
          const uint32_t left = nb - b;
          do_zero(rec, c0 + b, left < 4 ? left : 4, left < 4 && (left & 1), Live{});
          if (left == 1) {
            do_last(rec, c0 + b);
            continue;
          }
          do_pair(rec, c0 + b, Live{});
          if (left < 4) {
            if (left == 3) do_last(rec + PAIR_BYTES, c0 + b + 2);
            continue;
          }
          do_pair(rec + PAIR_BYTES, c0 + b + 2, Live{});
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[stage]);
      ready = __all_sync(0xffffffffu, ready);
      stage = next;
      if (next == 0) round++;
    }

    // ---- item epilogue: this warp's tiles are complete over the item's K range; write them out
    if (!dead && my_tile_exists) {
#pragma unroll
      for (int n = 0; n < NT; n++) {
        if (n > 0 && (uint32_t)n >= n_live) break;
        const uint32_t tok = n * 4 + t;
        const bool valid = tok < pcount;
        const uint32_t pair = valid ? s_pair[buf * 8 + tok] : 0;
        const float un = valid ? s_un[buf * 8 + tok] : 0.0f;
        const size_t row = (size_t)it.ks * n_pairs + pair;
#pragma unroll
        for (int j = 0; j < WARP_TILES; j++) {
          const uint32_t ptile = ITEM_TILES * tile + WARP_TILES * warp + j;  // packed tile index within the phase's region
          if (RAGGED && ptile >= packed_tiles) break;
          const float r_lo = (acc[j][n][0] + acc[j][n][1]) * un, r_hi = (acc[j][n][2] + acc[j][n][3]) * un;  // row slots g and g+8
          if (phase == 0) {
            // slots 0..7 of a gate/up tile are gate rows, slots 8..15 the matching up rows
            if (valid) {
              float *gp = p.parts + row * 2 * d.F + ptile * 8 + g;
              gp[0] = r_lo;
              gp[d.F] = r_hi;
            }
          } else if (valid) {
            float *yo = (k_is_split ? p.down_parts : d.y) + row * d.D + ptile * 16;
            yo[g] = r_lo;
            yo[g + 8] = r_hi;
          }
        }
      }
    }
  }
  if (cur_unit) leave_unit();
  if (dead && lane == 0) {
    *(volatile uint32_t *)s_abort = 1;
    atomicOr(d.status, MER_DEVSTAT_TIMEOUT);
  }
  if (!p.sync) continue;
  if (phase == 0) {
    // all partial sums, then all hidden rows
    if (LOCAL) {
      if (!grid_barrier(p.bar + 1, s_ok, d.status)) dead = true;
      if (threadIdx.x == 0) mbar_arrive(hidden);
      continue;
    }
    if (grid_barrier(p.bar + 1, s_ok, d.status)) {
      hidden_units(d, p.parts, p.ph[0].n_ksplit, p.ph[1], blockIdx.x, gridDim.x, warp, lane, s_red, reinterpret_cast<float4 *>(s_frag));
    } else {
      dead = true;
    }
    if (p.phases == 1) continue;  // the down phase is a launch of its own
    fence_async();
    if (!grid_barrier(p.bar + 2, s_ok, d.status)) dead = true;
    if (threadIdx.x == 0) mbar_arrive(hidden);
  } else if (p.tail != TAIL_NONE) {
    if (grid_barrier(p.bar + 3, s_ok, d.status) && !dead) ffn_stream_tail(p);
  }
  }
}

template <int DT, int NT, bool RAGGED, bool ROUTE, bool LOCAL>
__global__ void __launch_bounds__(THREADS, 1) k_ffn_stream(const __grid_constant__ StreamParams p) {
  ffn_stream_body<DT, NT, RAGGED, ROUTE, LOCAL>(p);
}

// The step between the phases as a kernel of its own, where a cooperative launch is refused.
__global__ void __launch_bounds__(CONSUMERS) k_hidden(const __grid_constant__ MoeDispatch d, const float *parts, uint32_t n_ksplit, const __grid_constant__ PhaseParams down) {
  extern __shared__ __align__(128) uint8_t smem[];  // 2 * CONSUMER_WARPS words, then the stash
  hidden_units(d, parts, n_ksplit, down, blockIdx.x, gridDim.x, threadIdx.x >> 5, threadIdx.x & 31, reinterpret_cast<uint32_t *>(smem), reinterpret_cast<float4 *>(smem + 128));
}

__global__ void __launch_bounds__(256) k_x_images(const __grid_constant__ MoeDispatch d) {
  __shared__ float s_max[8];
  build_wanted_image(d, blockIdx.x, s_max);
}

__global__ void k_reduce_ksplit(const float *__restrict__ part, float *__restrict__ y, size_t n, uint32_t n_ksplit) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float acc = part[i];
  for (uint32_t k = 1; k < n_ksplit; k++) acc += part[(size_t)k * n + i];
  y[i] = acc;
}

struct Plan {
  uint32_t nt, kc, n_stages, chunk_stride, n_frag, frag_cols, frag_bytes;
  PhaseParams ph[2];
  uint32_t queue[2];
  size_t smem;
};

constexpr size_t SMEM_LIMIT = 227 * 1024;
constexpr uint32_t MAX_KSPLIT = 64;

size_t frag_buffer(uint32_t kb_split, uint32_t cols) { return ((size_t)cols * (frag_stride(kb_split) + seed_words(kb_split) * 4) + 127) & ~(size_t)127; }

// The K split of one phase.  An item is 16 tiles (one per warp) over one split: multiples of 8 blocks, at least 16, within `max_ksplit`
// splits (what the partial-sum scratch can hold).  The one with the smallest estimated time of the busiest CTA is taken, in units of one
// block step (16 tiles x one block of K): a CTA gets its share of the items of kb_split block steps each and ends half an item behind the
// others (one or two items: the whole of it, as there is nothing to take over), and an item costs its switch, 800 cycles.  64 tokens on 128
// experts of 2048 x 768: 165 us a layer with splits of 32 and 24 blocks, 174 with 16 and 16, 168 with 64 and 24.
PhaseParams split_phase(int dtype, uint32_t kb_total, uint32_t packed_tiles, uint32_t cols, uint32_t active_groups, int n_ctas, uint32_t max_ksplit) {
  const uint32_t bb = dtype == MER_DTYPE_Q4_0 ? MER_Q4_BLOCK_BYTES : MER_Q8_BLOCK_BYTES;
  const uint32_t tile_groups = (packed_tiles + ITEM_TILES - 1) / ITEM_TILES;
  const uint64_t items_per_split = (uint64_t)active_groups * tile_groups;
  PhaseParams ph{packed_tiles, kb_total, kb_total, 1};
  const double per_item = dtype == MER_DTYPE_Q4_0 ? 5.0 : 3.0;
  double best = 1e30;
  uint32_t seen_split = 0;
  for (uint32_t n = 1; n <= max_ksplit; n++) {
    uint32_t split = ((kb_total + n - 1) / n + 7) / 8 * 8;
    if (split > kb_total) split = kb_total;
    if (n > 1 && split < 16) break;
    if (split == seen_split) continue;  // same split as a smaller n
    seen_split = split;
    const uint32_t nn = (kb_total + split - 1) / split;
    if (nn > max_ksplit) continue;
    // a ring of less than three stages of eight blocks loses more than a smaller split
    const uint32_t stage_blocks = split < 8 ? split : 8;
    if (HEADER_BYTES + frag_buffer(split, cols) + (size_t)3 * ITEM_TILES * stage_blocks * 16 * bb > SMEM_LIMIT && split > 16 && n < max_ksplit) continue;
    const uint64_t items = items_per_split * nn;
    const double per_cta = items <= 2 * (uint64_t)n_ctas ? (double)((items + n_ctas - 1) / n_ctas) : (double)items / n_ctas + 0.6;
    const double cost = per_cta * (split + per_item) + 0.5 * nn;  // last term: partial sums, and ties go to fewer splits
    if (cost < best) best = cost, ph.kb_split = split, ph.n_ksplit = nn;
  }
  return ph;
}

// Both phases of a dispatch.  Fragment arrays are sized by the most tokens any group can hold; there are two buffers of them if that leaves
// the ring 96 KB (what an SM streams in two microseconds).  A stage holds 8 (Q4_0) or 4 block pairs per warp if at least three stages
// then fit, else half of that, and so on (8: 2 % on one token).
Plan make_plan(int dtype, uint32_t D, uint32_t F, uint32_t nt, uint32_t max_group_tokens, uint32_t active_groups, int n_ctas, uint32_t cap_gate_up,
               uint32_t cap_down) {
  const uint32_t bb = dtype == MER_DTYPE_Q4_0 ? MER_Q4_BLOCK_BYTES : MER_Q8_BLOCK_BYTES;
  const uint32_t tp = 4 * nt, cols = 2 * (max_group_tokens < tp ? max_group_tokens : tp);
  const uint32_t cap[2] = {std::min(cap_gate_up, MAX_KSPLIT), std::min(cap_down, MAX_KSPLIT)};
  Plan pl{};
  pl.nt = nt, pl.frag_cols = cols;
  pl.ph[0] = split_phase(dtype, D / 32, F / 8, cols, active_groups, n_ctas, cap[0]);
  pl.ph[1] = split_phase(dtype, F / 32, (D + 15) / 16, cols, active_groups, n_ctas, cap[1]);
  for (;;) {
    const size_t frag = std::max(frag_buffer(pl.ph[0].kb_split, cols), frag_buffer(pl.ph[1].kb_split, cols));
    pl.frag_bytes = (uint32_t)frag;
    pl.n_frag = HEADER_BYTES + 2 * frag + (96u << 10) <= SMEM_LIMIT ? 2 : 1;
    const size_t fixed = HEADER_BYTES + pl.n_frag * frag;
    if (fixed < SMEM_LIMIT) {
      for (uint32_t ppw = dtype == MER_DTYPE_Q4_0 ? 8 : 4; ppw >= 1; ppw >>= 1) {
        pl.kc = std::min(2 * ppw, std::max(pl.ph[0].kb_split, pl.ph[1].kb_split));
        pl.chunk_stride = pl.kc * 16 * bb;
        const size_t stage = (size_t)ITEM_TILES * pl.chunk_stride;
        pl.n_stages = (uint32_t)std::min<size_t>(8, (SMEM_LIMIT - fixed) / stage);
        if (pl.n_stages >= 3 || (ppw == 1 && pl.n_stages >= 2)) {
          pl.smem = fixed + pl.n_stages * stage;
          for (int f = 0; f < 2; f++) pl.queue[f] = std::min(QUEUE, std::max(1u, (pl.n_stages * pl.kc + pl.ph[f].kb_split - 1) / pl.ph[f].kb_split));
          return pl;
        }
      }
    }
    // does not fit: halve the longer split (more partial sums) if the scratch allows
    const int f = frag_buffer(pl.ph[0].kb_split, cols) >= frag_buffer(pl.ph[1].kb_split, cols) ? 0 : 1;
    PhaseParams &ph = pl.ph[f];
    const uint32_t next_split = ((ph.kb_split + 1) / 2 + 7) / 8 * 8, next_n = (ph.kb_total + next_split - 1) / next_split;
    if (next_split >= ph.kb_split || next_split < 8 || next_n > cap[f]) {
      pl.n_stages = 0;
      return pl;
    }
    ph.kb_split = next_split, ph.n_ksplit = next_n;
  }
}

struct ScratchLayout {
  size_t bar, pos, npass, pgroup, pstart, pcount, pdesc, taken, bounds, seeds, x_un, h_un, parts, parts_bytes, total;
};

// `parts` holds the partial sums of whichever phase is running: gate/up partials [n_ksplit][P][2][F], then (after they have become hidden
// rows) down partials [n_ksplit][P][D].
ScratchLayout scratch_layout(uint32_t max_pairs, uint32_t D, uint32_t F) {
  ScratchLayout L{};
  size_t off = 0;
  auto take = [&](size_t bytes) {
    size_t o = off;
    off += (bytes + 255) & ~(size_t)255;
    return o;
  };
  L.bar = take(N_BARRIERS * 4);
  L.pos = take((size_t)max_pairs * 4);
  L.npass = take(256);
  L.pgroup = take(((size_t)std::max(max_pairs, 4096u) + 2) * 4);
  L.pstart = take((size_t)max_pairs * 4);
  L.pcount = take((size_t)max_pairs * 4);
  L.pdesc = take((size_t)max_pairs * sizeof(PassDesc));
  L.taken = take((size_t)2 * MER_MAX_CTAS1 * 8);
  L.bounds = take((size_t)2 * MER_MAX_CTAS1 * 4);
  L.seeds = take((size_t)max_pairs * 2 * image_seed_stride(std::max(D, F)) * 4);
  L.x_un = take((size_t)max_pairs * 4);
  // room for 8 splits of the largest batch, but never less than 64 splits of an 8-pair dispatch, capped at 1 GiB
  const size_t per_pair = (size_t)(2 * F > D ? 2 * F : D) * 4;
  size_t want = (size_t)8 * max_pairs * per_pair;
  const size_t small = (size_t)MAX_KSPLIT * 8 * per_pair;
  if (want < small) want = small;
  if (want > ((size_t)1 << 30)) want = (size_t)1 << 30;
  if (want < (size_t)max_pairs * per_pair) want = (size_t)max_pairs * per_pair;
  L.parts_bytes = want;
  L.h_un = take(std::max<size_t>(max_pairs, std::min((size_t)MAX_KSPLIT * max_pairs, want / ((size_t)D * 4))) * 4);  // of every pair and K split that the scratch can hold
  L.parts = take(want);
  L.total = off;
  return L;
}

template <int DT>
cudaError_t launch_stream(const StreamParams &p, uint32_t nt, bool local, size_t smem, int grid, cudaStream_t s) {
  bool ragged = p.kc % 4 != 0;
  for (const PhaseParams &ph : p.ph) ragged = ragged || ph.packed_tiles % ITEM_TILES != 0 || ph.kb_total % 4 != 0;
  auto one = [&](auto route, auto local) -> void (*)(StreamParams) {
    return ragged ? k_ffn_stream<DT, 1, true, decltype(route)::value, decltype(local)::value> : k_ffn_stream<DT, 1, false, decltype(route)::value, decltype(local)::value>;
  };
  using T = std::true_type;
  using F = std::false_type;
  void (*kern)(StreamParams) = nt == 2          ? (ragged ? k_ffn_stream<DT, 2, true, false, false> : k_ffn_stream<DT, 2, false, false, false>)
                               : p.d.route_here ? (local ? one(T{}, T{}) : one(T{}, F{}))
                                                : (local ? one(F{}, T{}) : one(F{}, F{}));
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  // the grid-wide steps wait for every CTA: a cooperative launch guarantees that they are all resident
  return launch_overlapped(kern, dim3(grid), THREADS, smem, s, p.sync != 0, p);
}

}  // namespace

bool stream_ffn_supported(int dtype, uint32_t D, uint32_t F) {
  if (dtype != MER_DTYPE_Q4_0 && dtype != MER_DTYPE_Q8_0) return false;
  if (D == 0 || F == 0 || D % 32 != 0 || F % 32 != 0) return false;  // rows of whole blocks: every tile chunk is a multiple of 16 bytes
  return make_plan(dtype, D, F, 1, 4, 1, 148, MAX_KSPLIT, MAX_KSPLIT).n_stages >= 2;
}

size_t stream_ffn_scratch_bytes(uint32_t max_pairs, uint32_t D, uint32_t F) { return scratch_layout(max_pairs, D, F).total; }

namespace {
// Token-pass width and plan of a dispatch (pure function of its shape and hints).
Plan plan_dispatch(const MoeDispatch &d, int sm_count) {
  const uint32_t P = d.n_tokens * d.slots;
  const ScratchLayout L = scratch_layout(d.scratch_pairs, d.D, d.F);
  const uint32_t mgt = d.max_group_tokens ? d.max_group_tokens : P, act = d.active_groups_hint ? d.active_groups_hint : 1;
  // how many K splits of partial sums the scratch can hold for this dispatch
  const uint32_t cap_gu = (uint32_t)std::min<size_t>(MAX_KSPLIT, L.parts_bytes / ((size_t)P * 2 * d.F * 4));
  const uint32_t cap_dn = (uint32_t)std::min<size_t>(MAX_KSPLIT, L.parts_bytes / ((size_t)P * d.D * 4));
  Plan pl = make_plan(d.dtype, d.D, d.F, mgt > 4 ? 2 : 1, mgt, act, sm_count, cap_gu, cap_dn);
  if (pl.nt == 2 && pl.n_stages < 3) pl = make_plan(d.dtype, d.D, d.F, 1, mgt, act, sm_count, cap_gu, cap_dn);  // eight tokens per pass do not fit: four
  return pl;
}
// At most one down item a CTA, of no more than one round of its warps (28 units, 3.5 rounds: one token on 8 experts of 4096 x 14336 209 us for
// 201), and room for both phases' partial sums: the kernels with LOCAL (one token on 128 experts of 2048 x 768 268 us for 284).
bool one_down_item(const MoeDispatch &d, const Plan &pl, size_t parts_bytes) {
  const uint64_t P = (uint64_t)d.n_tokens * d.slots;
  return pl.nt == 1 && P * d.items_per_pass[1] <= d.n_ctas && pl.frag_cols / 2 * ((pl.ph[1].kb_split + 3) / 4) <= CONSUMER_WARPS &&
         (pl.ph[0].n_ksplit * P * 2 * d.F + pl.ph[1].n_ksplit * P * d.D) * 4 <= parts_bytes;
}
}  // namespace

// (248 us for 268.  Where the weights of an item are longer it loses: one token on 8 experts of 4096 x 14336 208 us for 201.)
bool route_in_stream(const MoeDispatch &d, const RouterDev &r) {
  return d.pass_desc && d.x_rows && d.n_tokens == 1 && r.num_experts <= 256 && d.slots <= 32 &&
         one_down_item(d, plan_dispatch(d, (int)d.n_ctas), scratch_layout(d.scratch_pairs, d.D, d.F).parts_bytes);
}

void stream_bind(MoeDispatch &d, void *scratch, int sm_count, bool for_gemm) {
  if (sm_count > MER_MAX_CTAS1 - 1) sm_count = MER_MAX_CTAS1 - 1;
  uint8_t *base = static_cast<uint8_t *>(scratch);
  const ScratchLayout L = scratch_layout(d.scratch_pairs, d.D, d.F);
  d.n_passes = reinterpret_cast<uint32_t *>(base + L.npass);
  d.pass_group = reinterpret_cast<uint32_t *>(base + L.pgroup);
  d.pass_start = reinterpret_cast<uint32_t *>(base + L.pstart);
  d.pass_count = reinterpret_cast<uint32_t *>(base + L.pcount);
  d.pass_desc = reinterpret_cast<PassDesc *>(base + L.pdesc);
  d.taken = reinterpret_cast<uint64_t *>(base + L.taken);
  d.pos = for_gemm ? reinterpret_cast<uint32_t *>(base + L.pos) : nullptr;
  d.x_rows = d.y;  // [n_tokens x D] fp32 in size, and free until the down phase
  d.act_seeds = reinterpret_cast<float *>(base + L.seeds);
  d.x_un = reinterpret_cast<float *>(base + L.x_un);
  d.h_un = reinterpret_cast<float *>(base + L.h_un);
  const Plan pl = plan_dispatch(d, sm_count);
  d.tokens_per_pass = 4 * pl.nt;
  d.item_bounds = reinterpret_cast<uint32_t *>(base + L.bounds);
  for (int f = 0; f < 2; f++) d.items_per_pass[f] = pl.ph[f].n_ksplit * ((pl.ph[f].packed_tiles + ITEM_TILES - 1) / ITEM_TILES);
  d.n_ctas = (uint32_t)sm_count;
}

cudaError_t launch_ffn_stream(MoeDispatch &d, void *scratch, int sm_count, cudaStream_t s, int *launches, cudaEvent_t ev_mid) {
  if (sm_count > MER_MAX_CTAS1 - 1) sm_count = MER_MAX_CTAS1 - 1;  // the per-CTA work split holds at most 256 ranges
  const uint32_t P = d.n_tokens * d.slots;
  uint8_t *base = static_cast<uint8_t *>(scratch);
  const ScratchLayout L = scratch_layout(d.scratch_pairs, d.D, d.F);
  const Plan pl = plan_dispatch(d, sm_count);
  if (pl.n_stages < 2 || !d.pass_desc || d.tokens_per_pass != 4 * pl.nt) return cudaErrorInvalidConfiguration;
  StreamParams p{};
  p.d = d;
  p.ph[0] = pl.ph[0], p.ph[1] = pl.ph[1];
  p.kc = pl.kc, p.n_stages = pl.n_stages, p.chunk_stride = pl.chunk_stride;
  p.queue[0] = pl.queue[0], p.queue[1] = pl.queue[1];
  p.n_frag = pl.n_frag, p.frag_cols = pl.frag_cols, p.frag_bytes = pl.frag_bytes;
  p.parts = reinterpret_cast<float *>(base + L.parts);
  p.bar = reinterpret_cast<uint32_t *>(base + L.bar);
  const bool local = one_down_item(d, pl, L.parts_bytes);
  // the weighted combine of the layer rides on the same launch when the caller asked for it
  const int tail = d.fuse_combine ? TAIL_COMBINE : (d.fuse_reduce && pl.ph[1].n_ksplit > 1) ? TAIL_REDUCE : TAIL_NONE;
  cudaError_t e;
  int n = 0;
  auto launch = [&](uint32_t phases, bool sync) {
    const bool here = phases == 3 && sync && local;
    p.down_parts = here ? p.parts + (size_t)pl.ph[0].n_ksplit * P * 2 * d.F : p.parts;
    p.phases = phases, p.sync = sync ? 1 : 0, p.tail = sync && (phases & 2) ? tail : TAIL_NONE;
    n++;
    e = d.dtype == MER_DTYPE_Q4_0 ? launch_stream<MER_DTYPE_Q4_0>(p, pl.nt, here, pl.smem, sm_count, s) : launch_stream<MER_DTYPE_Q8_0>(p, pl.nt, here, pl.smem, sm_count, s);
    return e == cudaSuccess;
  };
  bool whole = true;  // the grid-wide steps ran
  if (ev_mid) {       // stage timers: a launch per phase
    if (!launch(1, true)) return e;
    cudaEventRecord(ev_mid, s);
    if (!launch(2, true)) return e;
  } else if (d.steps_apart || !launch(3, true)) {
    // a cooperative launch is refused: the steps between and behind the phases are kernels of their own
    cudaGetLastError();
    whole = false, n = 0;
    if (!launch(1, false)) return e;
    const uint32_t smem = 128 + pl.ph[1].kb_split * 128;
    if ((e = cudaFuncSetAttribute(k_hidden, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) != cudaSuccess) return e;
    k_hidden<<<std::min(P * pl.ph[1].n_ksplit, 8u * (uint32_t)sm_count), CONSUMERS, smem, s>>>(d, p.parts, pl.ph[0].n_ksplit, pl.ph[1]);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    n++;
    if (!launch(2, false)) return e;
  }
  d.combined = whole && tail == TAIL_COMBINE;
  // the per-pair outputs are the K-split partials until somebody adds them: the combine kernel does, or
  // launch_reduce_parts for entry points that return per-pair outputs
  d.y_parts = pl.ph[1].n_ksplit > 1 && !(whole && tail == TAIL_REDUCE) ? p.down_parts : nullptr;
  d.y_nparts = pl.ph[1].n_ksplit;
  if (launches) *launches += n;
  return cudaSuccess;
}

cudaError_t launch_x_images(const MoeDispatch &d, cudaStream_t s, int *launches) {
  if (!d.x_rows) return cudaSuccess;
  k_x_images<<<d.n_tokens, 256, 0, s>>>(d);
  if (launches) (*launches)++;
  return cudaGetLastError();
}

cudaError_t launch_reduce_parts(const MoeDispatch &d, cudaStream_t s, int *launches) {
  if (!d.y_parts || d.y_nparts <= 1) return cudaSuccess;
  size_t cnt = (size_t)d.n_tokens * d.slots * d.D;
  k_reduce_ksplit<<<(unsigned)((cnt + 255) / 256), 256, 0, s>>>(d.y_parts, d.y, cnt, d.y_nparts);
  if (launches) (*launches)++;
  return cudaGetLastError();
}
