// Router, token->expert grouping, generic (any-shape) expert FFN, combine, dequant dump.
//
// The generic FFN kernels are the slow, shape-agnostic path: one warp per output row, one
// weight per lane per step, fp32 FMA.  They handle rows that straddle blocks (d_model or
// d_ff not a multiple of 32, e.g. the reference's 37x45 test shape) and are the on-device
// cross-check for the streaming kernels.
#include "kernels.h"
#include "ptx.cuh"

#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>
#include <cfloat>

#include "../../include/mer_b200.h"
#include "act_image.cuh"
#include "layout.cuh"
#include "passes.cuh"
#include "route.cuh"

namespace {

__device__ __forceinline__ float f16_bits_to_f32(uint16_t v) { return __half2float(__ushort_as_half(v)); }

// One dequantised weight of a flat block stream: d * (q - 8) (Q4_0) or d * q (Q8_0); the
// product is exact in fp32 (11-bit significand times a <= 8-bit integer).
template <int DT>
__device__ __forceinline__ float decode_weight(const uint8_t *__restrict__ base, size_t flat) {
  size_t blk = flat >> 5;
  uint32_t j = (uint32_t)flat & 31u;
  if (DT == MER_DTYPE_Q8_0) {
    const uint8_t *b = base + blk * MER_Q8_BLOCK_BYTES;
    float d = f16_bits_to_f32(*reinterpret_cast<const uint16_t *>(b));
    return __fmul_rn(d, (float)(int8_t)b[2 + j]);
  } else {
    const uint8_t *b = base + blk * MER_Q4_BLOCK_BYTES;
    float d = f16_bits_to_f32(*reinterpret_cast<const uint16_t *>(b));
    uint32_t byte = b[2 + (j & 15u)];
    int q = (int)(j < 16u ? (byte & 15u) : (byte >> 4)) - 8;
    return __fmul_rn(d, (float)q);
  }
}

// Weight (matrix, row, col) of a resident expert in either slot layout.
template <int DT>
__device__ __forceinline__ float weight_at(const MoeDispatch &d, const uint8_t *__restrict__ base, int matrix, uint32_t row,
                                           uint32_t col) {
  if (d.packed) {
    PackedAddr a = packed_locate<DT>(d.D, d.F, matrix, row, col);
    float sc = f16_bits_to_f32(*reinterpret_cast<const uint16_t *>(base + a.scale));
    uint32_t byte = base[a.quant];
    int q = DT == MER_DTYPE_Q8_0 ? (int)byte - 128 : (int)((col & 16u) ? (byte >> 4) : (byte & 15u)) - 8;
    return __fmul_rn(sc, (float)q);
  }
  const size_t bb = DT == MER_DTYPE_Q8_0 ? MER_Q8_BLOCK_BYTES : MER_Q4_BLOCK_BYTES;
  const size_t proj = ((size_t)d.D * d.F + 31) / 32 * bb;
  const uint32_t K = matrix < 2 ? d.D : d.F;
  return decode_weight<DT>(base + (size_t)matrix * proj, (size_t)row * K + col);
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ float silu_f(float x) { return x / (1.0f + expf(-x)); }
__device__ __forceinline__ float clamp_gate(float g, float limit) {
  if (limit > 0.0f && isfinite(limit) && g == g) g = fminf(fmaxf(g, -limit), limit);  // NaN stays NaN
  return g;
}

// ---------------------------------------------------------------------------------------
// Router.  One CTA computes the logits of 1 to 8 experts for a tile of 4 tokens (every warp takes an
// eighth of the columns of all its rows, so W is read once per token tile and each lane has many
// independent loads in flight).  The last CTA to finish a token tile scores, filters and picks
// top-k for its tokens, one warp per token (LinearGate::route_with_scratch, gating.rs:395-476);
// the last tile overall groups the (token, slot) pairs by expert.
// ---------------------------------------------------------------------------------------
constexpr int ROUTER_THREADS = 256;
constexpr int ROUTER_WARPS = ROUTER_THREADS / 32;
constexpr int ROUTER_TT = 4;                      // tokens per CTA
constexpr uint32_t ROUTER_CTAS = 240;             // rows per CTA are halved while there are fewer CTAs than this
constexpr uint32_t SMALL_P = 4096;                // pair keys staged in shared memory below this many pairs
constexpr uint32_t STABLE_G = 512;                // (token, slot)-ordered grouping up to this many groups
constexpr int ROUTE_LATER = 3;                    // `group_here`: selection and grouping are the streaming kernel's
constexpr uint32_t GRID_GROUPING_PAIRS = 8192;    // from this many pairs the grouping runs grid-wide (count / scan / scatter)

// 64-bit divisions cost a few hundred cycles and much code, and this sits on the critical path of every decode layer: they are
// kept out of line, for sizes that need them.
__device__ __noinline__ uint32_t div64(uint64_t a, uint32_t b) { return (uint32_t)(a / b); }
// ceil(a * b / c)
__device__ __forceinline__ uint32_t scaled_ceil(uint32_t a, uint32_t b, uint32_t c) {
  const uint64_t v = (uint64_t)a * b + c - 1;
  return v <= 0xFFFFFFFFull ? (uint32_t)v / c : div64(v, c);
}
// ---- work split of the streaming kernels: one contiguous item range per CTA and phase.  An item of a pass with
// more than four tokens multiplies two token tiles instead of one: cost 13 vs 10.  (Gate/up of n passes of eight against 2n of
// four: 1.28 to 1.35 times the time a pass on Q8_0 experts of 4096 x 1536 and 2048 x 768, 1.36 and 1.42 on Q4_0 of 7168 x 2048 and 4096 x 14336.)
// `s_cum`: running cost before each pass and after the last, or null: all passes cost the same.  One CTA of 256 threads.
__device__ void build_item_bounds(const MoeDispatch &d, uint32_t n_passes, const uint32_t *s_cum) {
  const uint32_t G = d.n_ctas, i0 = d.items_per_pass[0], i1 = d.items_per_pass[1];
  const uint32_t total = s_cum ? s_cum[n_passes] : n_passes;  // at most 13 x 1024 weighted: products with G fit 32 bits
#pragma unroll 1
  for (uint32_t b = threadIdx.x; b <= G; b += 256) {
    uint32_t pass, b0, b1;  // first pass that is not wholly in front of the bound; items of it that are, in either phase
    if (s_cum) {
      const uint32_t target = total * b;
      uint32_t lo = 0, hi = n_passes;  // largest pass index with cum[pass] * G <= target
#pragma unroll 1
      while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (s_cum[mid] * G <= target) lo = mid; else hi = mid - 1;
      }
      pass = lo, b0 = b1 = 0;
      if (lo < n_passes) {
        const uint32_t w = s_cum[lo + 1] - s_cum[lo], wg = w * G, rem = target - s_cum[lo] * G;  // rem < wg
        b0 = scaled_ceil(rem, i0, wg), b1 = scaled_ceil(rem, i1, wg);
      }
    } else {
      const uint64_t target = (uint64_t)total * b;
      pass = target <= 0xFFFFFFFFull ? (uint32_t)target / G : div64(target, G);
      const uint32_t rem = (uint32_t)(target - (uint64_t)pass * G);
      b0 = scaled_ceil(rem, i0, G), b1 = scaled_ceil(rem, i1, G);
    }
    d.item_bounds[b] = pass * i0 + b0;
    d.item_bounds[MER_MAX_CTAS1 + b] = pass * i1 + b1;
  }
}

// Entry of the pass table.
__device__ __forceinline__ void put_pass(const MoeDispatch &d, uint32_t pass, uint32_t g, const uint8_t *base, uint32_t start, uint32_t count) {
  if (d.pass_desc) {
    d.pass_desc[pass].base = base, d.pass_desc[pass].count = count;
  } else {
    d.pass_group[pass] = g, d.pass_start[pass] = start, d.pass_count[pass] = count;
  }
}
__device__ __forceinline__ const uint8_t *expert_payload(const MoeDispatch &d, uint32_t eid) { return eid < d.max_experts ? d.expert_ptr[eid] : nullptr; }
__device__ __forceinline__ void put_pair(const MoeDispatch &d, uint32_t at, uint32_t pair) {
  d.perm[at] = pair;
  if (d.pos) d.pos[pair] = at;
}
__device__ __forceinline__ void clear_taken(const MoeDispatch &d) {  // by a CTA of 256 threads
  if (d.taken && threadIdx.x < d.n_ctas) d.taken[threadIdx.x] = 0, d.taken[MER_MAX_CTAS1 + threadIdx.x] = 0;
}

// Cuts every group into passes of at most d.tokens_per_pass pairs (the unit the streaming FFN works
// on).  One CTA of 256 threads; `off` = the group offsets.
// `perm_ready`: the pairs are in d.perm, else k_group_scatter puts them into the passes.
__device__ void build_passes_block(const MoeDispatch &d, const uint32_t *off, bool perm_ready) {
  __shared__ uint32_t s_pcnt[257];
  __shared__ uint8_t s_cost[1024];  // cost of each of the first 1024 passes (the weighted work split below)
  const uint32_t tpp = d.tokens_per_pass;
  const uint32_t tpp_shift = 31 - __clz(tpp);  // tokens per pass is a power of two (4 or 8; 128 or 256 for the GEMM kernels)
  clear_taken(d);
  const uint32_t per = (d.n_groups + 255) / 256;
  const uint32_t g0 = threadIdx.x * per, g1 = min(g0 + per, d.n_groups);
  uint32_t mine = 0;
#pragma unroll 1
  for (uint32_t g = g0; g < g1; g++) mine += (off[g + 1] - off[g] + tpp - 1) >> tpp_shift;
  s_pcnt[threadIdx.x + 1] = mine;
  if (threadIdx.x == 0) s_pcnt[0] = 0;
  __syncthreads();
  if (threadIdx.x < 32) {  // inclusive scan of 256 counts by one warp, 8 per lane
    uint32_t v[8], run = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) run += s_pcnt[1 + threadIdx.x * 8 + i], v[i] = run;
    uint32_t incl = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t up = __shfl_up_sync(0xffffffffu, incl, o);
      if (threadIdx.x >= (uint32_t)o) incl += up;
    }
    const uint32_t base = incl - run;
#pragma unroll
    for (int i = 0; i < 8; i++) s_pcnt[1 + threadIdx.x * 8 + i] = base + v[i];
  }
  __syncthreads();
  uint32_t np = s_pcnt[threadIdx.x];
#pragma unroll 1
  for (uint32_t g = g0; g < g1; g++) {
    const uint32_t beg = off[g], end = off[g + 1];
    const PassCut cut(end - beg, tpp, tpp_shift);
    const uint8_t *base = d.pass_desc && cut.passes ? expert_payload(d, d.group_expert[g]) : nullptr;
    uint32_t st = beg;
    if (d.pass_desc) d.pass_group[g] = np;
#pragma unroll 1
    for (uint32_t i = 0; i < cut.passes; i++) {
      const uint32_t cnt = cut.count(i, end - st);
      put_pass(d, np, g, base, st, cnt);
      if (d.pass_desc && perm_ready)
#pragma unroll 1
        for (uint32_t j = 0; j < cnt; j++) d.pass_desc[np].pair[j] = d.perm[st + j];
      if (np < 1024) s_cost[np] = cnt > 4 ? 13 : 10;
      np++, st += cnt;
    }
  }
  if (threadIdx.x == 0) d.n_passes[0] = s_pcnt[256];
  if (!d.item_bounds) return;
  __shared__ uint32_t s_cum[1025];
  const uint32_t n_passes = s_pcnt[256];
  __syncthreads();  // s_cost[] written above is read back below
  const bool weighted = n_passes <= 1024 && tpp == 8;
  if (weighted) {
    // inclusive scan of the pass costs: 4 per thread, then the same warp scan as above over the 256 partial sums
    uint32_t c[4], run = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint32_t q = threadIdx.x * 4 + i;
      c[i] = q < n_passes ? (uint32_t)s_cost[q] : 0u;
      run += c[i];
    }
    s_pcnt[threadIdx.x + 1] = run;
    __syncthreads();
    if (threadIdx.x < 32) {
      uint32_t v[8], r2 = 0;
#pragma unroll
      for (int i = 0; i < 8; i++) r2 += s_pcnt[1 + threadIdx.x * 8 + i], v[i] = r2;
      uint32_t incl = r2;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        uint32_t up = __shfl_up_sync(0xffffffffu, incl, o);
        if (threadIdx.x >= (uint32_t)o) incl += up;
      }
      const uint32_t base = incl - r2;
#pragma unroll
      for (int i = 0; i < 8; i++) s_pcnt[1 + threadIdx.x * 8 + i] = base + v[i];
    }
    __syncthreads();
    uint32_t acc = s_pcnt[threadIdx.x];  // cost of all passes before this thread's four
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint32_t q = threadIdx.x * 4 + i;
      if (q <= 1024) s_cum[q] = acc;
      acc += c[i];
    }
    if (threadIdx.x == 255) s_cum[1024] = acc;
    __syncthreads();
  }
  build_item_bounds(d, n_passes, weighted ? s_cum : nullptr);
}

// Group of pair p: local expert index, the shared-expert group, or MER_NONE for an unfilled / foreign slot.
__device__ __forceinline__ uint32_t pair_group_key(const RouterDev &r, const MoeDispatch &d, uint32_t p) {
  const uint32_t e = __ldcg(d.pair_expert + p);
  if (e == MER_NONE) return MER_NONE;
  if ((p % d.slots) >= r.top_k || e == r.shared_expert_id) return r.num_experts;  // shared-expert slot (or a dispatched row of it)
  return e - r.id_base;
}

// Grouping of a large dispatch in three grid-wide steps (count, scan, scatter) instead of one CTA.  The order of
// the pairs inside a group is whatever the atomics give; every pair's result is independent of its position.
__global__ void __launch_bounds__(256) k_group_count(RouterDev r, MoeDispatch d) {
  const uint32_t P = d.n_tokens * d.slots;
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < P; p += gridDim.x * blockDim.x) {
    const uint32_t k = pair_group_key(r, d, p);
    if (k != MER_NONE) atomicAdd(d.group_count + k, 1u);
  }
}
// `status`: where the router has left its bits, to be published (null: nothing to do).
__global__ void __launch_bounds__(256) k_group_scan(RouterDev r, MoeDispatch d, uint32_t *status) {
  if (status && threadIdx.x == 0) *d.status = atomicExch(status, 0u);
  const uint32_t G = d.n_groups;
  for (uint32_t g = threadIdx.x; g < G; g += blockDim.x) {
    d.group_expert[g] = (g < r.num_experts) ? r.id_base + g : r.shared_expert_id;
    d.group_cursor[g] = 0;  // of the scatter that follows
  }
  // the counts go through shared memory in slabs
  __shared__ uint32_t s_cnt[1024], s_warp[8];
  __shared__ uint32_t s_run;
  if (threadIdx.x == 0) s_run = 0;
  for (uint32_t g0 = 0; g0 < G; g0 += 1024) {
    const uint32_t n = min(1024u, G - g0);
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
      s_cnt[i] = d.group_count[g0 + i];
      d.group_count[g0 + i] = 0;  // zero again for the next dispatch's count
    }
    __syncthreads();
    {  // exclusive scan, four counts per thread
      uint32_t c[4], run = 0;
#pragma unroll
      for (uint32_t i = 0; i < 4; i++) c[i] = threadIdx.x * 4 + i < n ? s_cnt[threadIdx.x * 4 + i] : 0, run += c[i];
      uint32_t incl = run;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t up = __shfl_up_sync(0xffffffffu, incl, o);
        if ((threadIdx.x & 31) >= (uint32_t)o) incl += up;
      }
      if ((threadIdx.x & 31) == 31) s_warp[threadIdx.x >> 5] = incl;
      __syncthreads();
      uint32_t acc = s_run + incl - run, total = s_run;
#pragma unroll
      for (uint32_t w = 0; w < 8; w++) {
        if (w < threadIdx.x >> 5) acc += s_warp[w];
        total += s_warp[w];
      }
#pragma unroll
      for (uint32_t i = 0; i < 4; i++) {
        if (threadIdx.x * 4 + i < n) s_cnt[threadIdx.x * 4 + i] = acc;
        acc += c[i];
      }
      __syncthreads();
      if (threadIdx.x == 0) s_run = total;
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) d.offsets[g0 + i] = s_cnt[i];
  }
  __syncthreads();
  if (threadIdx.x == 0) d.offsets[G] = s_run;
  __threadfence_block();
  __syncthreads();
  if (d.pass_group) build_passes_block(d, d.offsets, false);
}
__global__ void __launch_bounds__(256) k_group_scatter(RouterDev r, MoeDispatch d) {
  const uint32_t P = d.n_tokens * d.slots;
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < P; p += gridDim.x * blockDim.x) {
    const uint32_t k = pair_group_key(r, d, p);
    if (k == MER_NONE) {
      if (d.pos) d.pos[p] = MER_NONE;
      continue;
    }
    const uint32_t rank = atomicAdd(d.group_cursor + k, 1u);
    put_pair(d, d.offsets[k] + rank, p);
    if (d.pass_desc) d.pass_desc[d.pass_group[k] + rank / d.tokens_per_pass].pair[rank % d.tokens_per_pass] = p;
  }
}
// Work split over passes of equal cost.
__device__ __forceinline__ void even_bounds(const MoeDispatch &d, uint32_t n_passes) {
  const uint32_t G = d.n_ctas, n0 = n_passes * d.items_per_pass[0], n1 = n_passes * d.items_per_pass[1];
  if (threadIdx.x <= G && (uint64_t)max(n0, n1) * G <= 0xFFFFFFFFull && G < 256) {
    d.item_bounds[threadIdx.x] = n0 * threadIdx.x / G;
    d.item_bounds[MER_MAX_CTAS1 + threadIdx.x] = n1 * threadIdx.x / G;
  } else if ((uint64_t)max(n0, n1) * G > 0xFFFFFFFFull || G >= 256) {
    build_item_bounds(d, n_passes, nullptr);
  }
}
// The same for at most 32 pairs of the streaming kernels, in registers of one warp: sorted position of every pair, the pairs
// that start a pass, their order.  The general form's dozen block-wide steps took 4 us on B200 for one token's eight pairs, as long
// as the kernels that follow need for the weights of half of them.
__device__ void build_groups_small(const RouterDev &r, const MoeDispatch &d) {
  __shared__ uint32_t s_np, s_cum[33];
  clear_taken(d);
  const uint32_t P = d.n_tokens * d.slots, tpp = d.tokens_per_pass;
  const bool weighted = tpp == 8;
  if (threadIdx.x < 32) {
    const uint32_t p = threadIdx.x, before = (1u << p) - 1;
    const uint32_t eid = p < P ? __ldcg(d.pair_expert + p) : MER_NONE;
    const uint8_t *base = expert_payload(d, eid);
    uint32_t key = eid;  // group index; unfilled slots sort last
    if (eid != MER_NONE) key = p % d.slots >= r.top_k || eid == r.shared_expert_id ? r.num_experts : eid - r.id_base;
    const uint32_t same = __match_any_sync(0xffffffffu, key), rank = __popc(same & before);
    uint32_t pos = rank;
#pragma unroll 4
    for (uint32_t j = 0; j < P; j++) pos += __shfl_sync(0xffffffffu, key, j) < key;
    const bool valid = key != MER_NONE, starts = valid && rank % tpp == 0;
    const uint32_t starters = __reduce_or_sync(0xffffffffu, starts ? 1u << pos : 0u);
    const uint32_t np = __popc(starters), n_valid = __popc(__ballot_sync(0xffffffffu, valid));
    if (valid) {
      d.perm[pos] = p;
      if (rank == 0) d.group_expert[key] = eid;
    }
    const uint32_t count = min(tpp, __popc(same) - rank), pass = __popc(starters & ((1u << pos) - 1));
    if (starts) put_pass(d, pass, key, base, pos, count);
    if (valid) d.pass_desc[__popc(starters & ((2u << pos) - 1)) - 1].pair[rank % tpp] = p;
    if (p == 0) {
      d.offsets[d.n_groups] = n_valid;  // all of the offsets that anyone reads after the streaming kernels
      d.n_passes[0] = s_np = np;
    }
    if (weighted) {
      if (starts) s_cum[pass + 1] = count > 4 ? 13 : 10;
      __syncwarp();
      uint32_t incl = p < np ? s_cum[p + 1] : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t up = __shfl_up_sync(0xffffffffu, incl, o);
        if (p >= (uint32_t)o) incl += up;
      }
      s_cum[p + 1] = incl;
      if (p == 0) s_cum[0] = 0;
    }
  }
  __syncthreads();
  if (weighted) return build_item_bounds(d, s_np, s_cum);
  even_bounds(d, s_np);
}
// The same for the pairs of one token, at most 32: every pair that has an expert is a pass of its own.  `eid`: expert of pair threadIdx.x (first warp).
__device__ __forceinline__ void build_groups_token(const MoeDispatch &d, uint32_t eid) {
  __shared__ uint32_t s_np;
  clear_taken(d);
  if (threadIdx.x < 32) {
    const uint32_t p = threadIdx.x;
    const uint32_t valid = __ballot_sync(0xffffffffu, eid != MER_NONE), pass = __popc(valid & ((1u << p) - 1));
    if (eid != MER_NONE) {
      put_pass(d, pass, 0, expert_payload(d, eid), pass, 1);
      d.pass_desc[pass].pair[0] = p;
      d.perm[pass] = p;
    }
    if (p == 0) d.offsets[d.n_groups] = d.n_passes[0] = s_np = __popc(valid);
  }
  __syncthreads();
  even_bounds(d, s_np);
}

// The same for a batch of decode size (at most 2048 pairs, 512 groups): the counting atomics hand out the pairs' ranks, and
// one scan of packed counts gives every group its first pair, its first pass and the cost of the passes before it.  The order of
// the pairs inside a group is whatever the atomics give; every pair's result is independent of its position.  (The
// general form: a dozen more block-wide steps, 7 us for 512 pairs of 128 groups.)
constexpr uint32_t MID_PAIRS = 2048, MID_GROUPS = 512;
// `s_pair` [P]: group (16 bits) and rank of every pair.  Loops stay rolled: the code runs once, cold.
__device__ void build_groups_mid(const RouterDev &r, const MoeDispatch &d, uint32_t *s_pair) {
  constexpr uint32_t PER_G = MID_GROUPS / 256;
  __shared__ uint32_t s_cnt[MID_GROUPS], s_pass[MID_GROUPS], s_cum[MID_PAIRS / 8 + MID_GROUPS + 1];  // s_cum: passes of eight
  __shared__ uint64_t s_part[8];
  const uint32_t P = d.n_tokens * d.slots, G = d.n_groups, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t tpp = d.tokens_per_pass, shift = 31 - __clz(tpp);
  const bool bounds = d.item_bounds != nullptr, weighted = bounds && tpp == 8;  // (passes of four can be more than s_cum holds)
  for (uint32_t i = tid; i < MID_GROUPS; i += 256) s_cnt[i] = 0;
  clear_taken(d);
  // the payloads of the thread's groups: a round trip that passes while the pairs are counted
  const uint8_t *payload[PER_G];
#pragma unroll
  for (uint32_t i = 0; i < PER_G; i++) {
    const uint32_t g = tid * PER_G + i;
    payload[i] = d.pass_desc && g < G ? expert_payload(d, g < r.num_experts ? r.id_base + g : r.shared_expert_id) : nullptr;
  }
  __syncthreads();
#pragma unroll 1
  for (uint32_t p0 = tid; p0 < P; p0 += 512) {  // two loads in flight
    uint32_t eid[2];
#pragma unroll
    for (uint32_t i = 0; i < 2; i++) eid[i] = p0 + i * 256 < P ? __ldcg(d.pair_expert + p0 + i * 256) : MER_NONE;
#pragma unroll
    for (uint32_t i = 0; i < 2; i++) {
      const uint32_t p = p0 + i * 256;
      if (p >= P) break;
      uint32_t v = MER_NONE;
      if (eid[i] != MER_NONE) {
        const uint32_t key = eid[i] == r.shared_expert_id || p % d.slots >= r.top_k ? r.num_experts : eid[i] - r.id_base;
        v = key << 16 | atomicAdd(&s_cnt[key], 1u);
      }
      s_pair[p] = v;
    }
  }
  __syncthreads();
  // packed: pairs (20 bits), passes (20 bits), cost; thread t owns groups t * PER_G ..
  const auto packed = [&](uint32_t n) -> uint64_t {
    const uint32_t full = n >> shift, rest = n & (tpp - 1);
    const uint32_t cost = full * (tpp > 4 ? 13 : 10) + (rest == 0 ? 0 : rest > 4 ? 13 : 10);
    return n | (uint64_t)(full + (rest != 0)) << 20 | (uint64_t)cost << 40;
  };
  uint64_t mine[PER_G], run = 0;
#pragma unroll
  for (uint32_t i = 0; i < PER_G; i++) mine[i] = packed(s_cnt[tid * PER_G + i]), run += mine[i];
  uint64_t incl = run;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint64_t up = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= (uint32_t)o) incl += up;
  }
  if (lane == 31) s_part[warp] = incl;
  __syncthreads();
  uint64_t base = incl - run, total = 0;
#pragma unroll
  for (uint32_t w = 0; w < 8; w++) {
    if (w < warp) base += s_part[w];
    total += s_part[w];
  }
  const uint32_t n_passes = (uint32_t)(total >> 20) & 0xFFFFF;
#pragma unroll
  for (uint32_t i = 0; i < PER_G; i++) {
    const uint32_t g = tid * PER_G + i, n = (uint32_t)mine[i] & 0xFFFFF, beg = (uint32_t)base & 0xFFFFF;
    uint32_t pass = (uint32_t)(base >> 20) & 0xFFFFF, cum = (uint32_t)(base >> 40);
    s_cnt[g] = beg, s_pass[g] = pass;
    if (g < G) {
      const uint32_t eid = g < r.num_experts ? r.id_base + g : r.shared_expert_id;
      d.group_expert[g] = eid;
      d.offsets[g] = beg;
      const PassCut cut(n, tpp, shift);
      uint32_t st = 0;
#pragma unroll 1
      for (uint32_t j = 0; j < cut.passes; j++, pass++) {
        const uint32_t cnt = cut.count(j, n - st);
        put_pass(d, pass, g, payload[i], beg + st, cnt);
        st += cnt;
        if (weighted) s_cum[pass] = cum, cum += cnt > 4 ? 13 : 10;
      }
    }
    base += mine[i];
  }
  if (tid == 0) {
    d.offsets[G] = (uint32_t)total & 0xFFFFF;
    d.n_passes[0] = n_passes;
    if (weighted) s_cum[n_passes] = (uint32_t)(total >> 40);
  }
  __syncthreads();
#pragma unroll 1
  for (uint32_t p = tid; p < P; p += 256) {
    const uint32_t v = s_pair[p];
    if (v == MER_NONE) {
      if (d.pos) d.pos[p] = MER_NONE;
      continue;
    }
    const uint32_t g = v >> 16, rank = v & 0xFFFF;
    put_pair(d, s_cnt[g] + rank, p);
    if (d.pass_desc) d.pass_desc[s_pass[g] + (rank >> shift)].pair[rank & (tpp - 1)] = p;
  }
  if (bounds) build_item_bounds(d, n_passes, weighted ? s_cum : nullptr);
}

// Runs in one CTA after every token has been routed: groups pairs by expert.
__device__ void build_groups_layer(const RouterDev &r, const MoeDispatch &d, uint32_t *s_u32) {
  const uint32_t P = d.n_tokens * d.slots;
  if (P <= 32 && d.item_bounds) return build_groups_small(r, d);
  if (P <= MID_PAIRS && d.n_groups <= MID_GROUPS && d.pass_group) return build_groups_mid(r, d, s_u32);
  const uint32_t G = d.n_groups;
  const uint32_t tid = threadIdx.x, nt = blockDim.x, warp = tid >> 5, lane = tid & 31;
  uint32_t *s_off = s_u32;                    // [G + 1]
  uint32_t *s_cnt = s_u32 + G + 1;            // [8 warps][G] (stable path) or [G]
  const bool stable = G <= STABLE_G;
  uint32_t *s_key = s_cnt + (stable ? ROUTER_WARPS * G : G);  // [min(P, SMALL_P)]
  const bool staged = P <= SMALL_P;
  auto key_global = [&](uint32_t p) -> uint32_t {
    uint32_t e = __ldcg(d.pair_expert + p);
    if (e == MER_NONE) return MER_NONE;
    if ((p % d.slots) >= r.top_k || e == r.shared_expert_id) return r.num_experts;  // shared-expert slot (or a dispatched row of it)
    return e - r.id_base;
  };
  auto key_of = [&](uint32_t p) -> uint32_t { return staged ? s_key[p] : key_global(p); };
#pragma unroll 1
  for (uint32_t g = tid; g < G; g += nt) d.group_expert[g] = (g < r.num_experts) ? r.id_base + g : r.shared_expert_id;
#pragma unroll 1
  for (uint32_t i = tid; i < (stable ? ROUTER_WARPS * G : G); i += nt) s_cnt[i] = 0;
  if (staged)
#pragma unroll 1
    for (uint32_t p = tid; p < P; p += nt) s_key[p] = key_global(p);
  __syncthreads();
  if (stable) {
    // every warp owns a contiguous run of pairs, so (warp, position in run) order = (token, slot) order
    const uint32_t chunk = ((P + ROUTER_WARPS - 1) / ROUTER_WARPS + 31) / 32 * 32;
    const uint32_t p0 = warp * chunk, p1 = min(P, p0 + chunk);
#pragma unroll 1
    for (uint32_t p = p0 + lane; p < p1; p += 32) {
      uint32_t k = key_of(p);
      if (k != MER_NONE) atomicAdd(&s_cnt[warp * G + k], 1u);
    }
    __syncthreads();
#pragma unroll 1
    for (uint32_t g = tid; g < G; g += nt) {  // per group: exclusive scan over the warps, total into s_off
      uint32_t run = 0;
#pragma unroll 1
      for (uint32_t w = 0; w < ROUTER_WARPS; w++) {
        uint32_t c = s_cnt[w * G + g];
        s_cnt[w * G + g] = run;
        run += c;
      }
      s_off[g] = run;
    }
    __syncthreads();
    if (warp == 0) {  // exclusive scan of the group totals
      const uint32_t per = (G + 31) / 32;
      uint32_t run = 0;
#pragma unroll 1
      for (uint32_t i = 0; i < per; i++) {
        uint32_t g = lane * per + i;
        if (g < G) run += s_off[g];
      }
      uint32_t incl = run;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        uint32_t up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += up;
      }
      uint32_t base = incl - run;
#pragma unroll 1
      for (uint32_t i = 0; i < per; i++) {
        uint32_t g = lane * per + i;
        if (g < G) {
          uint32_t c = s_off[g];
          s_off[g] = base;
          base += c;
        }
      }
      if (lane == 31) s_off[G] = incl;
    }
    __syncthreads();
#pragma unroll 1
    for (uint32_t pb = p0; pb < p1; pb += 32) {
      const uint32_t p = pb + lane;
      const uint32_t k = p < p1 ? key_of(p) : MER_NONE;
      const uint32_t same = __match_any_sync(0xffffffffu, k);
      if (k != MER_NONE) {
        const uint32_t rank = __popc(same & ((1u << lane) - 1));
        put_pair(d, s_off[k] + s_cnt[warp * G + k] + rank, p);
      } else if (d.pos && p < p1) {
        d.pos[p] = MER_NONE;
      }
      __syncwarp();
      if (k != MER_NONE && (same & ((1u << lane) - 1)) == 0) s_cnt[warp * G + k] += __popc(same);
      __syncwarp();
    }
  } else {
#pragma unroll 1
    for (uint32_t p = tid; p < P; p += nt) {
      uint32_t k = key_of(p);
      if (k != MER_NONE) atomicAdd(&s_cnt[k], 1u);
    }
    __syncthreads();
    if (tid == 0) {
      uint32_t acc = 0;
#pragma unroll 1
      for (uint32_t g = 0; g < G; g++) {
        s_off[g] = acc;
        acc += s_cnt[g];
        s_cnt[g] = 0;
      }
      s_off[G] = acc;
    }
    __syncthreads();
#pragma unroll 1
    for (uint32_t p = tid; p < P; p += nt) {
      uint32_t k = key_of(p);
      if (k != MER_NONE) put_pair(d, s_off[k] + atomicAdd(&s_cnt[k], 1u), p);
      else if (d.pos) d.pos[p] = MER_NONE;
    }
  }
  __syncthreads();
#pragma unroll 1
  for (uint32_t g = tid; g <= G; g += nt) d.offsets[g] = s_off[g];
  if (d.pass_group) build_passes_block(d, s_off, true);
}

// A large dispatch is grouped by grid-wide kernels; their count step is done here, over the CTA's tokens first (an atomic per pick: all of a
// batch's on a few cache lines, 2048 tokens 16 us of selection instead of 13).  Out of line: small calls run past it cold.
__device__ __noinline__ void count_picks(const RouterDev &r, const MoeDispatch &d, uint32_t picked, uint32_t tokens, uint32_t *s_hist) {
  const uint32_t E = r.num_experts;
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < E; i += ROUTER_THREADS) s_hist[i] = 0;
  __syncthreads();
  if (picked != MER_NONE) atomicAdd(&s_hist[picked], 1u);
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < E; i += ROUTER_THREADS)
    if (s_hist[i]) atomicAdd(d.group_count + i, s_hist[i]);
  if (threadIdx.x == 0 && d.slots > r.top_k) atomicAdd(d.group_count + E, tokens);
}

// Selection for the TT tokens from t0 on, whose logits are there, one warp per token; the last of `n_tiles` CTAs that get here groups all pairs.
// `direct`: the logits [TT][stride] in shared memory, or null: in d.logits, with PARTS as `sets` partial sums ([sets][T][E], added in order).
// EJ > 0: at most 32 EJ experts and 32 pairs of the streaming kernels, with no other code in the kernel: it runs once a layer, cold, and what a call of one
// token waits for is its instructions (one token on 128 experts of 2048 x 768: 1 us a layer).
template <int TT, int EJ, bool PARTS>
__device__ __forceinline__ void finish_tokens(const RouterDev &r, const MoeDispatch &d, uint32_t t0, uint32_t n_tiles, const float *direct, uint32_t stride, uint32_t sets,
                                              bool recheck, uint8_t *smem_raw, uint32_t *status, uint32_t max_tokens, int group_here) {
  const uint32_t E = r.num_experts, D = d.D, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __shared__ uint32_t s_last;
  __shared__ uint32_t s_groups[TT][64];
  __shared__ float s_gscore[TT][64];
  uint32_t picked = MER_NONE;
  if (warp < min((uint32_t)TT, d.n_tokens - t0)) {
    float *s_score = reinterpret_cast<float *>(smem_raw) + (size_t)warp * 2 * E;  // [E] scores (become mixing weights)
    float *s_sel = s_score + E;                                                    // [E] selection scores
    uint8_t *s_ok = smem_raw + (size_t)TT * 2 * E * 4 + (size_t)warp * E;          // [E] allowed & not yet taken
    const uint32_t token = t0 + warp;
    bool bad = false;
    // The loads of a row are in flight together (one by one, a round trip to L2 per 32 experts: 3 us of 256).  Up to 32 experts have one value a lane: there
    // AHEAD partial sums are (set by set, 4097 tokens on 8 experts of 512 x 512 94.3 us a layer instead of 88.5, 600 on 32 of 7168 173.5 instead of 171).
    auto gather = [&](auto batch_tag, auto ahead_tag) {
      constexpr int BATCH = decltype(batch_tag)::value;
#pragma unroll 1
      for (uint32_t i0 = lane; i0 < E; i0 += 32 * BATCH) {
        float v[BATCH];
#pragma unroll
        for (int j = 0; j < BATCH; j++) {
          const uint32_t i = i0 + 32 * j;
          v[j] = i >= E ? 0.0f : direct ? direct[warp * stride + i] : __ldcg(d.logits + (size_t)token * E + i);
        }
        if constexpr (PARTS) {
          constexpr int AHEAD = decltype(ahead_tag)::value;
#pragma unroll 1
          for (uint32_t z0 = 1; z0 < sets; z0 += AHEAD) {
            float part[AHEAD][BATCH];
#pragma unroll
            for (int z = 0; z < AHEAD; z++)
#pragma unroll
              for (int j = 0; j < BATCH; j++)
                part[z][j] = z0 + z < sets && i0 + 32 * j < E ? __ldcg(d.logits + ((size_t)(z0 + z) * d.n_tokens + token) * E + i0 + 32 * j) : 0.0f;
#pragma unroll
            for (int z = 0; z < AHEAD; z++)
#pragma unroll
              for (int j = 0; j < BATCH; j++)
                if (z0 + z < sets) v[j] += part[z][j];
          }
        }
#pragma unroll
        for (int j = 0; j < BATCH; j++) {
          if (i0 + 32 * j < E) s_score[i0 + 32 * j] = v[j];
          bad |= !(fabsf(v[j]) <= FLT_MAX);
        }
      }
    };
    if (PARTS && E <= 32)
      gather(std::integral_constant<int, 1>{}, std::integral_constant<int, 4>{});
    else
      gather(std::integral_constant<int, EJ == 0 ? 8 : EJ>{}, std::integral_constant<int, 1>{});
    // Non-finite values do not survive the split into parts (kernels_logits.cu): such a token's logits are made again in fp32.
    if (recheck && __any_sync(0xffffffffu, bad))
#pragma unroll 1
      for (uint32_t e = 0; e < E; e++) {
        float v = 0.0f;
        for (uint32_t i = lane; i < D; i += 32) v = fmaf(__ldg(r.w + (size_t)e * D + i), __ldg(d.x + (size_t)token * D + i), v);
        v = warp_sum(v);
        if (lane == 0) s_score[e] = v;
      }
    __syncwarp();
    Pick pick;
    if constexpr (EJ > 0)
      pick = route_token_reg<EJ>(r, s_score, s_sel, status);
    else
      pick = route_token(r, s_score, s_sel, s_ok, s_groups[warp], s_gscore[warp], status);
    const size_t p0 = (size_t)token * d.slots;
    if (lane < r.top_k) picked = pick.id;
    if (lane < r.top_k) {
      d.pair_expert[p0 + lane] = pick.id == MER_NONE ? MER_NONE : r.id_base + pick.id;
      d.pair_weight[p0 + lane] = pick.weight;
    }
    if (lane == 0 && d.slots > r.top_k) {
      d.pair_expert[p0 + r.top_k] = r.shared_expert_id;
      d.pair_weight[p0 + r.top_k] = r.shared_scale ? r.shared_scale[token] : 1.0f;
    }
  }
  if (EJ == 0 && group_here == 2) return count_picks(r, d, picked, min((uint32_t)TT, d.n_tokens - t0), reinterpret_cast<uint32_t *>(smem_raw));
  if (group_here != 1) return;
  __syncthreads();
  if (n_tiles > 1) {
    if (threadIdx.x == 0) {
      const uint32_t prev = arrive_acq_rel(&d.counters[max_tokens]);
      s_last = (prev == n_tiles - 1);
      if (s_last) d.counters[max_tokens] = 0;
    }
    __syncthreads();
    if (!s_last) return;
  }
  if constexpr (EJ > 0) {
    if (d.n_tokens == 1) {  // the picks are still in the first warp's registers
      const uint32_t eid = threadIdx.x < r.top_k ? (picked == MER_NONE ? MER_NONE : r.id_base + picked) : threadIdx.x < d.slots ? r.shared_expert_id : MER_NONE;
      build_groups_token(d, eid);
    } else {
      build_groups_small(r, d);
    }
  } else {
    build_groups_layer(r, d, reinterpret_cast<uint32_t *>(smem_raw));
  }
  if (threadIdx.x == 0) *d.status = atomicExch(status, 0u);  // (a round trip that nobody waits for here)
}

template <int ROWS, int EJ>
__global__ void __launch_bounds__(ROUTER_THREADS) k_router(RouterDev r, MoeDispatch d, uint32_t max_tokens, int group_here, uint32_t logit_ctas) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  const uint32_t E = r.num_experts, D = d.D;
  const uint32_t tile = blockIdx.y, t0 = tile * ROUTER_TT;
  const uint32_t n_here = min((uint32_t)ROUTER_TT, d.n_tokens - t0);
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t e0 = blockIdx.x * ROWS;
  __shared__ float s_part[ROWS][ROUTER_TT][ROUTER_WARPS + 1];  // [row][token][warp]
  __shared__ float s_logit[ROUTER_TT][ROWS];                  // used when one CTA covers all experts
  const bool single = logit_ctas == 1 && group_here != ROUTE_LATER;
  // Status bits gather in a scratch word, which the grouping publishes: no launch clears them.
  uint32_t *const status = group_here ? d.counters + max_tokens + 1 : d.status;
  // What the steps behind the logits read once a layer, and the layers in between have long pushed out of L2: a miss each, on their
  // critical path.
  if (tile == 0 && warp == 1) {
    const uint32_t line = 128 / 4 * (blockIdx.x * 32 + lane);  // a CTA covers 32 lines
    if (line < E) {
      if (r.logit_bias) prefetch_l2(r.logit_bias + line);
      if (r.correction_bias) prefetch_l2(r.correction_bias + line);
    }
    if (d.pass_desc && line / 2 < E && r.id_base + line / 2 < d.max_experts) prefetch_l2(d.expert_ptr + r.id_base + line / 2);
  }
  // And the router's weights, which nothing before this kernel writes: behind the norm kernel the CTAs wait here for 4 us.
  if (tile == 0 && blockIdx.x < logit_ctas && e0 < E) {
    const float *rows = r.w + (size_t)e0 * D;
    for (uint32_t i = threadIdx.x * 32; i < min((uint32_t)ROWS, E - e0) * D; i += ROUTER_THREADS * 32) prefetch_l2(rows + i);
  }
  grid_dep_wait();
  grid_dep_launch();

  if (blockIdx.x >= logit_ctas) {  // CTAs beside the logits' make the activation images of the tile's tokens
    const uint32_t tt = blockIdx.x - logit_ctas;
    if (group_here == ROUTE_LATER && tt == 0) {  // what the grouping would clear
      if (threadIdx.x == 0) *d.status = 0;
      clear_taken(d);
    }
    if (tt < n_here) build_x_image(d, t0 + tt, threadIdx.x, ROUTER_THREADS, &s_part[0][0][0]);
    return;
  }
  // Rows of whole groups of 32 values: a slice of D / 32 groups of four for each warp, whatever that is (a warp per expert row with single loads, one token after the
  // other: 16 tokens on 64 experts of 2816 x 1536 106 us a layer instead of 98, 7 on 16 of 736 x 992 33 instead of 30).
  if ((D & 31u) == 0) {
    const uint32_t slice4 = D / 4 / ROUTER_WARPS;  // float4 per warp slice
    float acc[ROWS][ROUTER_TT];
#pragma unroll
    for (int rr = 0; rr < ROWS; rr++)
#pragma unroll
      for (int tt = 0; tt < ROUTER_TT; tt++) acc[rr][tt] = 0.0f;
#pragma unroll (ROWS >= 8 ? 2 : 4)
    for (uint32_t i = lane; i < slice4; i += 32) {
      float4 b[ROUTER_TT], a[ROWS];
#pragma unroll
      for (int tt = 0; tt < ROUTER_TT; tt++) {
        b[tt] = make_float4(0, 0, 0, 0);
        if ((uint32_t)tt < n_here) b[tt] = __ldg(reinterpret_cast<const float4 *>(d.x + (size_t)(t0 + tt) * D) + warp * slice4 + i);
      }
#pragma unroll
      for (int rr = 0; rr < ROWS; rr++) {
        const uint32_t row = min(e0 + rr, E - 1);
        a[rr] = __ldg(reinterpret_cast<const float4 *>(r.w + (size_t)row * D) + warp * slice4 + i);
      }
#pragma unroll
      for (int rr = 0; rr < ROWS; rr++)
#pragma unroll
        for (int tt = 0; tt < ROUTER_TT; tt++) {
          acc[rr][tt] = fmaf(a[rr].x, b[tt].x, acc[rr][tt]);
          acc[rr][tt] = fmaf(a[rr].y, b[tt].y, acc[rr][tt]);
          acc[rr][tt] = fmaf(a[rr].z, b[tt].z, acc[rr][tt]);
          acc[rr][tt] = fmaf(a[rr].w, b[tt].w, acc[rr][tt]);
        }
    }
    // Sums over the warp: in each step a lane hands on half of its values, so that it ends with the sum of one (31 shuffles for 32 values instead
    // of 160; the additions are those of warp_sum).
    constexpr int N = ROWS * ROUTER_TT;
    float v[N];
#pragma unroll
    for (int i = 0; i < N; i++) v[i] = acc[i / ROUTER_TT][i % ROUTER_TT];
    uint32_t at = 0;
#pragma unroll
    for (int step = 0; step < 5; step++) {
      const int o = 16 >> step, n = N >> (step + 1);
      const bool upper = lane & o;
#pragma unroll
      for (int i = 0; i < N / 2; i++)
        if (i < n) {
          const float other = __shfl_xor_sync(0xffffffffu, upper ? v[i] : v[n + i], o);
          v[i] = (upper ? v[n + i] : v[i]) + other;
        }
      if (n > 0)
        at += upper ? n : 0;
      else
        v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    }
    if ((lane & (32 / N - 1)) == 0) (&s_part[0][0][0])[at * (ROUTER_WARPS + 1) + warp] = v[0];
    __syncthreads();
    if (threadIdx.x < ROWS * ROUTER_TT) {
      const uint32_t rr = threadIdx.x / ROUTER_TT, tt = threadIdx.x % ROUTER_TT;
      float v = 0.0f;
#pragma unroll
      for (int w = 0; w < ROUTER_WARPS; w++) v += s_part[rr][tt][w];
      if (single)
        s_logit[tt][rr] = v;
      else if (e0 + rr < E && tt < n_here)
        d.logits[(size_t)(t0 + tt) * E + e0 + rr] = v;
    }
  } else {
    // any d_model: warp = expert row, tokens one after the other
    const uint32_t e = warp < ROWS ? e0 + warp : E;
    for (uint32_t tt = 0; tt < n_here; tt++) {
      float acc = 0.0f;
      if (e < E) {
        const float *w = r.w + (size_t)e * D, *x = d.x + (size_t)(t0 + tt) * D;
        for (uint32_t i = lane; i < D; i += 32) acc = fmaf(__ldg(w + i), __ldg(x + i), acc);
        acc = warp_sum(acc);
      }
      if (lane == 0 && e < E) {
        if (single)
          s_logit[tt][warp] = acc;
        else
          d.logits[(size_t)(t0 + tt) * E + e] = acc;
      }
    }
  }
  if (group_here == ROUTE_LATER) return;
  __shared__ uint32_t s_flag;
  __syncthreads();
  if (!single) {
    if (threadIdx.x == 0) {
      const uint32_t prev = arrive_acq_rel(&d.counters[tile]);
      s_flag = (prev == logit_ctas - 1);
      if (s_flag) d.counters[tile] = 0;  // re-arm for the next launch
    }
    __syncthreads();
    if (!s_flag) return;
  }

  // ---- this CTA holds the last logits of the token tile
  finish_tokens<ROUTER_TT, EJ, false>(r, d, t0, gridDim.y, single ? &s_logit[0][0] : nullptr, ROWS, 1, false, smem_raw, status, max_tokens, group_here);
}

// The same behind the logits kernel of a large batch: every warp has a token.  (In the kernel above, whose registers leave room for two CTAs on an SM,
// 4096 tokens of 256 experts took 47 us.)
template <int TT>
__global__ void __launch_bounds__(ROUTER_THREADS) k_router_select(const __grid_constant__ RouterDev r, const __grid_constant__ MoeDispatch d, uint32_t max_tokens, uint32_t sets,
                                                                  int recheck, int group_here, uint32_t select_ctas) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  if (blockIdx.x >= select_ctas) {  // activation images of the tokens
    build_x_image(d, blockIdx.x - select_ctas, threadIdx.x, ROUTER_THREADS, reinterpret_cast<float *>(smem_raw));
    return;
  }
  uint32_t *const status = group_here ? d.counters + max_tokens + 1 : d.status;
  finish_tokens<TT, 0, true>(r, d, blockIdx.x * TT, select_ctas, nullptr, 0, sets, recheck != 0, smem_raw, status, max_tokens, group_here);
}

// Routing of a whole layer supplied by the caller (pair_expert already filled): group by expert.  The first CTA; the others make the activation images.
__global__ void __launch_bounds__(ROUTER_THREADS) k_groups_layer(RouterDev r, MoeDispatch d) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  if (blockIdx.x > 0) {
    __shared__ float s_max[ROUTER_WARPS];
    return build_wanted_image(d, blockIdx.x - 1, s_max);
  }
  build_groups_layer(r, d, reinterpret_cast<uint32_t *>(smem_raw));
}

// Routing supplied by the caller: mode 0 = every pair is its own group, mode 1 = one group.
// The first CTA; the others make the tokens' activation images.
__global__ void __launch_bounds__(256) k_groups_from_pairs(const __grid_constant__ MoeDispatch d, int single_group) {
  grid_dep_wait();
  grid_dep_launch();
  if (blockIdx.x > 0) {
    __shared__ float s_max[8];
    build_x_image(d, blockIdx.x - 1, threadIdx.x, 256, s_max);
    return;
  }
  const uint32_t P = d.n_tokens * d.slots;
  if (!single_group && d.pass_desc && d.n_tokens == 1) {
    if (threadIdx.x == 0) *d.status = 0;
    build_groups_token(d, threadIdx.x < P ? d.pair_expert[threadIdx.x] : MER_NONE);
    return;
  }
  for (uint32_t p = threadIdx.x; p < P; p += blockDim.x) {
    put_pair(d, p, p);
    if (!single_group) {
      d.group_expert[p] = d.pair_expert[p];
      d.offsets[p] = p;
    }
  }
  if (threadIdx.x == 0) {
    *d.status = 0;
    if (single_group) {
      d.group_expert[0] = d.pair_expert[0];
      d.offsets[0] = 0;
      d.offsets[1] = P;
    } else {
      d.offsets[P] = P;
    }
  }
  if (d.pass_group) {
    __syncthreads();  // the offsets written above are read back by the whole block
    build_passes_block(d, d.offsets, true);
  }
}

// ---------------------------------------------------------------------------------------
// Generic expert FFN.
// ---------------------------------------------------------------------------------------
constexpr int GEN_TG = 4;  // tokens of a group handled per pass over a weight row

__device__ __forceinline__ const uint8_t *group_weights(const MoeDispatch &d, uint32_t g) {
  uint32_t eid = d.group_expert[g];
  const uint8_t *base = (eid < d.max_experts) ? d.expert_ptr[eid] : nullptr;
  if (!base && threadIdx.x == 0) atomicOr(d.status, MER_DEVSTAT_RESIDENCY_MISS);
  return base;
}

template <int DT>
__global__ void __launch_bounds__(256) k_gate_up_generic(MoeDispatch d) {
  const uint32_t g = blockIdx.y;
  const uint32_t beg = d.offsets[g], end = d.offsets[g + 1];
  if (beg == end) return;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t r = blockIdx.x * 8 + warp;
  const uint8_t *base = group_weights(d, g);
  if (r >= d.F) return;
  if (!base) {  // fail closed: the pair contributes zeros and the host reports the miss
    for (uint32_t t = beg + lane; t < end; t += 32) d.h[(size_t)d.perm[t] * d.F + r] = 0.0f;
    return;
  }
  for (uint32_t t0 = beg; t0 < end; t0 += GEN_TG) {
    uint32_t pair[GEN_TG];
    const float *xs[GEN_TG];
    float ag[GEN_TG], au[GEN_TG];
#pragma unroll
    for (int t = 0; t < GEN_TG; t++) {
      pair[t] = (t0 + t < end) ? d.perm[t0 + t] : MER_NONE;
      xs[t] = d.x + (size_t)(pair[t] == MER_NONE ? 0 : pair[t] / d.slots) * d.D;
      ag[t] = au[t] = 0.0f;
    }
    for (uint32_t c = lane; c < d.D; c += 32) {
      float wg = weight_at<DT>(d, base, 0, r, c), wu = weight_at<DT>(d, base, 1, r, c);
#pragma unroll
      for (int t = 0; t < GEN_TG; t++) {
        float xv = __ldg(xs[t] + c);
        ag[t] = fmaf(wg, xv, ag[t]);
        au[t] = fmaf(wu, xv, au[t]);
      }
    }
#pragma unroll
    for (int t = 0; t < GEN_TG; t++) {
      float gsum = warp_sum(ag[t]), usum = warp_sum(au[t]);
      if (lane == 0 && pair[t] != MER_NONE)
        d.h[(size_t)pair[t] * d.F + r] = silu_f(clamp_gate(gsum, d.swiglu_limit)) * usum;
    }
  }
}

template <int DT>
__global__ void __launch_bounds__(256) k_down_generic(MoeDispatch d) {
  const uint32_t g = blockIdx.y;
  const uint32_t beg = d.offsets[g], end = d.offsets[g + 1];
  if (beg == end) return;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t r = blockIdx.x * 8 + warp;
  const uint8_t *base = group_weights(d, g);  // latches the residency miss: the slot may have gone since gate/up ran
  if (r >= d.D) return;
  if (!base) {
    for (uint32_t t = beg + lane; t < end; t += 32) d.y[(size_t)d.perm[t] * d.D + r] = 0.0f;
    return;
  }
  for (uint32_t t0 = beg; t0 < end; t0 += GEN_TG) {
    uint32_t pair[GEN_TG];
    const float *hs[GEN_TG];
    float acc[GEN_TG];
#pragma unroll
    for (int t = 0; t < GEN_TG; t++) {
      pair[t] = (t0 + t < end) ? d.perm[t0 + t] : MER_NONE;
      hs[t] = d.h + (size_t)(pair[t] == MER_NONE ? d.perm[beg] : pair[t]) * d.F;
      acc[t] = 0.0f;
    }
    for (uint32_t c = lane; c < d.F; c += 32) {
      float w = weight_at<DT>(d, base, 2, r, c);
#pragma unroll
      for (int t = 0; t < GEN_TG; t++) acc[t] = fmaf(w, hs[t][c], acc[t]);
    }
#pragma unroll
    for (int t = 0; t < GEN_TG; t++) {
      float s = warp_sum(acc[t]);
      if (lane == 0 && pair[t] != MER_NONE) d.y[(size_t)pair[t] * d.D + r] = s;
    }
  }
}

// out[token] = sum over slots, in slot order, of weight * y (combine_outputs_into,
// inference.rs:4472-4491; zero weights and unfilled slots skipped as engine.rs:5575-5581).
// Multiply and add round separately, as the reference's `*dst += weight * *v` does.
__global__ void __launch_bounds__(256) k_combine(MoeDispatch d) {
  const uint32_t token = blockIdx.y;
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.D) return;
  float acc = 0.0f;
  for (uint32_t s = 0; s < d.slots; s++) {
    if (d.residual && s == d.routed_slots) acc = __fadd_rn(d.residual[(size_t)token * d.D + i], acc);  // hidden + routed sum
    size_t p = (size_t)token * d.slots + s;
    float w = d.pair_weight[p];
    if (d.pair_expert[p] == MER_NONE || w == 0.0f) continue;
    float yv;
    if (d.y_parts && d.y_nparts > 1) {  // the streaming FFN left K-split partials: add them in split order
      const size_t n = (size_t)d.n_tokens * d.slots * d.D;
      yv = d.y_parts[p * d.D + i];
#pragma unroll 8
      for (uint32_t k = 1; k < d.y_nparts; k++) yv += d.y_parts[(size_t)k * n + p * d.D + i];
    } else {
      yv = d.y[p * d.D + i];
    }
    acc = __fadd_rn(acc, __fmul_rn(w, yv));
  }
  if (d.residual && d.routed_slots >= d.slots) acc = __fadd_rn(d.residual[(size_t)token * d.D + i], acc);
  d.out[(size_t)token * d.D + i] = acc;
}

// The same sum for final per-pair outputs (no K-split partials) and d_model % 4 == 0: one CTA per token, a thread four
// consecutive values; the rows of eight slots are loaded before the first is consumed (the one-value-per-thread form
// above moved 150 MB at 3 TB/s on a 2048-token batch).  Order and rounding are unchanged.
__global__ void __launch_bounds__(256) k_combine_rows4(MoeDispatch d) {
  const uint32_t token = blockIdx.x, S = d.slots;
  __shared__ float s_w[64];
  if (threadIdx.x < S && threadIdx.x < 64) {
    const size_t p = (size_t)token * S + threadIdx.x;
    const float w = d.pair_weight[p];
    s_w[threadIdx.x] = d.pair_expert[p] == MER_NONE ? 0.0f : w;  // a zero weight skips the slot
  }
  __syncthreads();
  const float4 *y4 = reinterpret_cast<const float4 *>(d.y) + (size_t)token * S * (d.D / 4);
  const float4 *res4 = d.residual ? reinterpret_cast<const float4 *>(d.residual) + (size_t)token * (d.D / 4) : nullptr;
  for (uint32_t i4 = threadIdx.x; i4 < d.D / 4; i4 += blockDim.x) {
    float4 acc = make_float4(0, 0, 0, 0);
    for (uint32_t s0 = 0; s0 <= S; s0 += 8) {
      float4 y[8];
#pragma unroll
      for (int j = 0; j < 8; j++)
        y[j] = (s0 + j < S && s_w[s0 + j] != 0.0f) ? __ldcs(y4 + (size_t)(s0 + j) * (d.D / 4) + i4) : make_float4(0, 0, 0, 0);
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const uint32_t sl = s0 + j;
        if (sl > S) break;
        if (res4 && sl == min(d.routed_slots, S)) {  // hidden + routed sum, before the shared expert's slot
          const float4 r = __ldg(res4 + i4);
          acc.x = __fadd_rn(r.x, acc.x), acc.y = __fadd_rn(r.y, acc.y), acc.z = __fadd_rn(r.z, acc.z), acc.w = __fadd_rn(r.w, acc.w);
        }
        if (sl == S) continue;
        const float wt = s_w[sl];
        if (wt == 0.0f) continue;
        acc.x = __fadd_rn(acc.x, __fmul_rn(wt, y[j].x));
        acc.y = __fadd_rn(acc.y, __fmul_rn(wt, y[j].y));
        acc.z = __fadd_rn(acc.z, __fmul_rn(wt, y[j].z));
        acc.w = __fadd_rn(acc.w, __fmul_rn(wt, y[j].w));
      }
    }
    reinterpret_cast<float4 *>(d.out)[(size_t)token * (d.D / 4) + i4] = acc;
  }
}

// A few KB between pinned host memory and the device, as kernels of the call's own sequence: a copy node waits 3 to 4 us for the copy
// engine on either side.  `status` (may be null) is cleared on the way in; on the way out `done` is written last, for a host
// that polls it.
constexpr int HOST_COPY_THREADS = 1024;
__global__ void __launch_bounds__(HOST_COPY_THREADS) k_host_in(const uint32_t *__restrict__ src, uint32_t *__restrict__ dst, uint32_t n, uint32_t *status) {
  grid_dep_launch();
  if (blockIdx.x == 0 && threadIdx.x == 0 && status) *status = 0;
  const uint32_t n4 = n / 4, i = blockIdx.x * HOST_COPY_THREADS + threadIdx.x;
  if (i < n4) reinterpret_cast<uint4 *>(dst)[i] = reinterpret_cast<const uint4 *>(src)[i];
  if (i < n % 4) dst[n4 * 4 + i] = src[n4 * 4 + i];
}
__global__ void __launch_bounds__(HOST_COPY_THREADS) k_host_out(const uint32_t *src, uint32_t stride, uint32_t rows, uint32_t n, uint32_t *dst, uint32_t *count,
                                                                uint32_t *done) {
  grid_dep_wait();
  for (uint32_t r = 0; r < rows; r++)
    for (uint32_t i = threadIdx.x; i < n; i += HOST_COPY_THREADS) dst[r * n + i] = __ldcg(src + (size_t)r * stride + i);
  if (!done) return;
  __threadfence_system();
  __syncthreads();
  if (threadIdx.x == 0) *(volatile uint32_t *)done = ++*count;
}

// RMSNorm of every token row and / or the shared expert's gate scalar (RmsNorm::forward_inplace, transformer.rs:62-74;
// SharedExpert::forward, transformer.rs:2224-2231).  One CTA per token; sums are block tree reductions (the
// reference adds left to right: rounding differs in the last bits only).
constexpr int PRE_THREADS = 512;
// VEC: D is a multiple of four and the rows are read and written four values at a time (16 tokens of 7168: 5 us, 18 us one by one).
template <bool VEC>
__global__ void __launch_bounds__(PRE_THREADS) k_pre_moe(const float *__restrict__ x, uint32_t D, const float *__restrict__ rms_weight, float eps,
                                                         const float *__restrict__ shared_gate, float *__restrict__ xn,
                                                         float *__restrict__ shared_scale) {
  constexpr int W = VEC ? 4 : 1;
  __shared__ float s_red[2][PRE_THREADS / 32];
  const uint32_t token = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n = D / W;
  const float *row = x + (size_t)token * D;
  auto load = [](const float *p, uint32_t i, float (&v)[W]) {
    if (VEC) {
      const float4 q = __ldg(reinterpret_cast<const float4 *>(p) + i);
      v[0] = q.x, v[1 % W] = q.y, v[2 % W] = q.z, v[3 % W] = q.w;
    } else {
      v[0] = __ldg(p + i);
    }
  };
  auto block_sum = [&](float v, int k) -> float {
    v = warp_sum(v);
    if (lane == 0) s_red[k][warp] = v;
    __syncthreads();
    float t = 0.0f;
#pragma unroll
    for (int w = 0; w < PRE_THREADS / 32; w++) t += s_red[k][w];
    return t;
  };
  float scale = 1.0f;
  grid_dep_wait();
  grid_dep_launch();
  if (rms_weight) {
    float sq = 0.0f;
#pragma unroll 4
    for (uint32_t i = threadIdx.x; i < n; i += PRE_THREADS) {
      float v[W];
      load(row, i, v);
#pragma unroll
      for (int j = 0; j < W; j++) sq = fmaf(v[j], v[j], sq);
    }
    sq = block_sum(sq, 0);
    scale = 1.0f / sqrtf(sq / (float)D + eps);
  }
  float dot = 0.0f;
#pragma unroll 4
  for (uint32_t i = threadIdx.x; i < n; i += PRE_THREADS) {
    float v[W], g[W];
    load(row, i, v);
    if (rms_weight) {
      load(rms_weight, i, g);
#pragma unroll
      for (int j = 0; j < W; j++) v[j] = __fmul_rn(__fmul_rn(v[j], scale), g[j]);  // x * scale * weight, rounded after each product
      float *dst = xn + (size_t)token * D + (size_t)i * W;
      if (VEC)
        *reinterpret_cast<float4 *>(dst) = make_float4(v[0], v[1 % W], v[2 % W], v[3 % W]);
      else
        *dst = v[0];
    }
    if (shared_gate) {
      load(shared_gate, i, g);
#pragma unroll
      for (int j = 0; j < W; j++) dot = fmaf(g[j], v[j], dot);
    }
  }
  if (shared_gate) {
    dot = block_sum(dot, 1);
    if (threadIdx.x == 0) shared_scale[token] = 1.0f / (1.0f + expf(-dot));
  }
}

template <int DT>
__global__ void k_dequant(const uint8_t *__restrict__ src, float *__restrict__ dst, size_t n) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  size_t stride = (size_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) dst[i] = decode_weight<DT>(src, i);
}

template <int DT>
__global__ void k_dequant_packed(const uint8_t *__restrict__ expert, int matrix, uint32_t D, uint32_t F, float *__restrict__ dst) {
  const uint32_t rows = matrix < 2 ? F : D, cols = matrix < 2 ? D : F;
  size_t n = (size_t)rows * cols;
  size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    uint32_t row = (uint32_t)(i / cols), col = (uint32_t)(i % cols);
    PackedAddr a = packed_locate<DT>(D, F, matrix, row, col);
    float sc = f16_bits_to_f32(*reinterpret_cast<const uint16_t *>(expert + a.scale));
    uint32_t byte = expert[a.quant];
    int q = DT == MER_DTYPE_Q8_0 ? (int)byte - 128 : (int)((col & 16u) ? (byte >> 4) : (byte & 15u)) - 8;
    dst[i] = __fmul_rn(sc, (float)q);
  }
}

__device__ __forceinline__ void write_slot(const SlotWrite &sw) {
  if (sw.slot) *reinterpret_cast<SlotHeader *>(sw.slot) = SlotHeader{sw.epoch, sw.expert_id, sw.dtype, sw.payload_bytes};
  *sw.entry = sw.payload;
}
__global__ void k_slot_write(SlotWrite sw) { write_slot(sw); }

// One thread per source block: copies its scale and its quant bytes to their packed places.
template <int DT>
__global__ void k_repack(const uint8_t *__restrict__ flat, uint8_t *__restrict__ packed, uint32_t D, uint32_t F, SlotWrite sw) {
  if (blockIdx.x == 0 && threadIdx.x == 0) write_slot(sw);  // readers wait for the event behind this kernel
  constexpr uint32_t BB = DT == MER_DTYPE_Q8_0 ? MER_Q8_BLOCK_BYTES : MER_Q4_BLOCK_BYTES;
  const size_t per_matrix = (size_t)D * F / 32;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < 3 * per_matrix; i += stride) {
    const int matrix = (int)(i / per_matrix);
    const size_t blk = i % per_matrix;
    const uint32_t K = matrix < 2 ? D : F;
    const uint32_t row = (uint32_t)(blk / (K / 32)), kb = (uint32_t)(blk % (K / 32));
    const uint16_t *src = reinterpret_cast<const uint16_t *>(flat + i * BB);  // blocks are 2-byte aligned
    PackedAddr a0 = packed_locate<DT>(D, F, matrix, row, kb * 32);
    *reinterpret_cast<uint16_t *>(packed + a0.scale) = src[0];
    if (DT == MER_DTYPE_Q4_0) {
#pragma unroll
      for (uint32_t t = 0; t < 4; t++) {  // quant bytes 4t..4t+3 hold elements 4t.. (low) and 16+4t.. (high)
        PackedAddr a = packed_locate<DT>(D, F, matrix, row, kb * 32 + 4 * t);
        *reinterpret_cast<uint32_t *>(packed + a.quant) = (uint32_t)src[1 + 2 * t] | ((uint32_t)src[2 + 2 * t] << 16);
      }
    } else {
#pragma unroll
      for (uint32_t t = 0; t < 4; t++) {
        PackedAddr a = packed_locate<DT>(D, F, matrix, row, kb * 32 + 8 * t);
        uint2 v;
        v.x = (uint32_t)src[1 + 4 * t] | ((uint32_t)src[2 + 4 * t] << 16);
        v.y = (uint32_t)src[3 + 4 * t] | ((uint32_t)src[4 + 4 * t] << 16);
        v.x ^= 0x80808080u, v.y ^= 0x80808080u;  // q + 128
        *reinterpret_cast<uint2 *>(packed + a.quant) = v;
      }
    }
  }
}

// Raw block-stream matvec for the qualification cases: one warp per row.
template <int DT>
__global__ void k_raw_matvec(const uint8_t *__restrict__ w, const float *__restrict__ x, float *__restrict__ y, size_t rows,
                             size_t cols) {
  size_t r = (size_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  uint32_t lane = threadIdx.x & 31;
  if (r >= rows) return;
  float acc = 0.0f;
  for (size_t c = lane; c < cols; c += 32) acc = fmaf(decode_weight<DT>(w, r * cols + c), x[c], acc);
  acc = warp_sum(acc);
  if (lane == 0) y[r] = acc;
}

__global__ void k_f16_to_f32(const uint16_t *__restrict__ src, float *__restrict__ dst, size_t n) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = f16_bits_to_f32(src[i]);
}
__global__ void k_f32_to_f16(const float *__restrict__ src, uint16_t *__restrict__ dst, size_t n) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = __half_as_ushort(__float2half_rn(src[i]));
}

// A kernel's dynamic shared memory needs leave where it and the kernel's own tables are more than 48 KB together; the routing and grouping kernels have up to 18 KB of
// tables.  (Asked for from 48 KB of dynamic memory on, calls of 438 to 682 experts and 256 tokens, or of 900 to 1365 and a few, failed to launch.)
constexpr size_t TABLE_BYTES = 20 * 1024;
template <class Kernel>
cudaError_t allow_smem(Kernel kern, size_t smem) {
  return smem + TABLE_BYTES > 48 * 1024 ? cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) : cudaSuccess;
}

}  // namespace


cudaError_t launch_router(const RouterDev &r, const MoeDispatch &d, uint32_t max_tokens, cudaStream_t s,
                          int *launches, bool group) {
  const uint32_t E = r.num_experts, G = d.n_groups;
  const uint32_t P = d.n_tokens * d.slots;
  const size_t smem_grp = (size_t)(G + 1 + (G <= STABLE_G ? ROUTER_WARPS * G : G) + (P <= SMALL_P ? P : 0)) * 4;
  const bool grid_grouping = group && P >= GRID_GROUPING_PAIRS && d.group_count != nullptr;
  const int group_here = group && d.route_here ? ROUTE_LATER : grid_grouping ? 2 : group ? 1 : 0;
  auto room = [&](auto kern, uint32_t tokens, size_t &smem) -> cudaError_t {
    smem = (std::max((size_t)tokens * E * 9, group_here == 1 ? smem_grp : (size_t)0) + 15) & ~(size_t)15;
    return allow_smem(kern, smem);
  };
  size_t smem;
  cudaError_t e;
  // From a few hundred tokens the logits are a GEMM of their own, unless the experts are so few that most of a tile would be
  // padding (8 experts, 256 tokens of 4096: 19 us of logits kernel).  Up to 16 experts, rows of whole 1024 values never go there.  Others did while the vector code
  // took whole 1024 only; now those go that are more than VECTOR_CTAS of its CTAs.  Us a layer, GEMM / vector, 8 experts and 256 tokens of 2816 63 / 52, of 7936 139 / 91,
  // 8 and 2048 (512 CTAs) of 1280 97 / 87, of 6400 239 / 214, 16 and 1024 (512) of 1280 80 / 68, of 5376 143 / 141; beyond the line 8 and 2900 (725) of 1280 116 / 123, of
  // 5376 280 / 285, 16 and 2048 (1024) of 1280 103 / 103, 8 and 4096 (1024) of 512 72 / 78.  The vector code's weights are the nearer to 64 bits (rms 0.7 to 2.1e-7 for
  // 0.8 to 2.5e-7).
  constexpr uint32_t VECTOR_CTAS = 512;
  const uint64_t vector_ctas = (uint64_t)((E + 7) / 8) * ((d.n_tokens + ROUTER_TT - 1) / ROUTER_TT);
  if (d.n_tokens >= 256 && d.D % 256 == 0 && (E > 16 || (d.D % 1024 != 0 && vector_ctas > VECTOR_CTAS))) {
    uint32_t sets = 1;
    bool in_parts = false;
    if ((e = launch_router_logits(r, d, group_here ? d.counters + max_tokens + 1 : d.status, &sets, &in_parts, s)) != cudaSuccess) return e;
    const uint32_t tokens = E <= 2048 ? ROUTER_WARPS : ROUTER_WARPS / 2;  // what fits shared memory
    auto kern = E <= 2048 ? k_router_select<ROUTER_WARPS> : k_router_select<ROUTER_WARPS / 2>;
    if ((e = room(kern, tokens, smem)) != cudaSuccess) return e;
    const uint32_t ctas = (d.n_tokens + tokens - 1) / tokens;
    kern<<<ctas + (d.x_rows ? d.n_tokens : 0), ROUTER_THREADS, smem, s>>>(r, d, max_tokens, sets, in_parts ? 1 : 0, group_here, ctas);
    e = cudaGetLastError();
    if (launches) (*launches)++;
  } else {
    // Expert rows per CTA: eight share the loads of x best, but a small call wants its few rows on as many SMs as there are
    // (one token, 128 experts of 2048: 13.4 us with a row per CTA, 16.6 us with eight).
    const uint32_t tiles = (d.n_tokens + ROUTER_TT - 1) / ROUTER_TT;
    uint32_t rows = 8;
    while (rows > 1 && d.D % 32 == 0 && (E + rows - 1) / rows * tiles < ROUTER_CTAS) rows >>= 1;
    const uint32_t logit_ctas = (E + rows - 1) / rows;
    const dim3 grid(logit_ctas + (d.x_rows ? ROUTER_TT : 0), tiles);
    auto kern = rows == 1 ? k_router<1, 0> : rows == 2 ? k_router<2, 0> : rows == 4 ? k_router<4, 0> : k_router<8, 0>;
    if ((group_here == 1 || group_here == ROUTE_LATER) && P <= 32 && d.item_bounds && E <= 256)
      kern = E <= 128 ? (rows == 1 ? k_router<1, 4> : rows == 2 ? k_router<2, 4> : rows == 4 ? k_router<4, 4> : k_router<8, 4>)
                      : (rows == 1 ? k_router<1, 8> : rows == 2 ? k_router<2, 8> : rows == 4 ? k_router<4, 8> : k_router<8, 8>);
    if ((e = room(kern, ROUTER_TT, smem)) != cudaSuccess) return e;
    e = launch_overlapped(kern, grid, ROUTER_THREADS, smem, s, false, r, d, max_tokens, group_here, logit_ctas);
  }
  if (e != cudaSuccess) return e;
  if (launches) (*launches)++;
  if (grid_grouping) {  // the router has counted the pairs per group
    const unsigned blocks = (P + 1023) / 1024;
    k_group_scan<<<1, 256, 0, s>>>(r, d, d.counters + max_tokens + 1);
    k_group_scatter<<<blocks, 256, 0, s>>>(r, d);
    if (launches) (*launches) += 2;
  }
  return cudaGetLastError();
}

bool groups_layer_on_grid(const MoeDispatch &d) { return d.n_tokens * d.slots >= GRID_GROUPING_PAIRS && d.group_count != nullptr; }

cudaError_t launch_groups_layer(const RouterDev &r, const MoeDispatch &d, cudaStream_t s, int *launches, bool counted) {
  const uint32_t G = d.n_groups, P = d.n_tokens * d.slots;
  if (groups_layer_on_grid(d)) {  // a large dispatch: count / scan / scatter over the grid
    const unsigned blocks = (P + 1023) / 1024;
    if (!counted) k_group_count<<<blocks, 256, 0, s>>>(r, d);
    k_group_scan<<<1, 256, 0, s>>>(r, d, nullptr);
    k_group_scatter<<<blocks, 256, 0, s>>>(r, d);
    if (launches) (*launches) += counted ? 2 : 3;
    return launch_x_images(d, s, launches);
  }
  size_t smem = (size_t)(G + 1 + (G <= STABLE_G ? ROUTER_WARPS * G : G) + (P <= SMALL_P ? P : 0)) * 4;
  smem = (smem + 15) & ~(size_t)15;
  const cudaError_t e = allow_smem(k_groups_layer, smem);
  if (e != cudaSuccess) return e;
  k_groups_layer<<<d.x_rows ? 1 + d.n_tokens : 1, ROUTER_THREADS, smem, s>>>(r, d);
  if (launches) (*launches)++;
  return cudaGetLastError();
}

cudaError_t launch_groups_from_pairs(const MoeDispatch &d, cudaStream_t s, int *launches) {
  const cudaError_t e = launch_overlapped(k_groups_from_pairs, dim3(d.x_rows ? 1 + d.n_tokens : 1), 256, 0, s, false, d, d.n_groups == 1);
  if (launches) (*launches)++;
  return e;
}

cudaError_t launch_ffn_generic(const MoeDispatch &d, cudaStream_t s, int *launches, cudaEvent_t ev_mid) {
  dim3 g1((d.F + 7) / 8, d.n_groups), g2((d.D + 7) / 8, d.n_groups);
  if (d.dtype == MER_DTYPE_Q8_0) {
    k_gate_up_generic<MER_DTYPE_Q8_0><<<g1, 256, 0, s>>>(d);
    if (ev_mid) cudaEventRecord(ev_mid, s);
    k_down_generic<MER_DTYPE_Q8_0><<<g2, 256, 0, s>>>(d);
  } else {
    k_gate_up_generic<MER_DTYPE_Q4_0><<<g1, 256, 0, s>>>(d);
    if (ev_mid) cudaEventRecord(ev_mid, s);
    k_down_generic<MER_DTYPE_Q4_0><<<g2, 256, 0, s>>>(d);
  }
  if (launches) (*launches) += 2;
  return cudaGetLastError();
}

cudaError_t launch_combine(const MoeDispatch &d, cudaStream_t s, int *launches) {
  if (d.combined) return cudaSuccess;  // the expert FFN launch already did it
  if (!(d.y_parts && d.y_nparts > 1) && (d.D & 3u) == 0 && d.slots <= 64) {
    k_combine_rows4<<<d.n_tokens, 256, 0, s>>>(d);
  } else {
    dim3 grid((d.D + 255) / 256, d.n_tokens);
    k_combine<<<grid, 256, 0, s>>>(d);
  }
  if (launches) (*launches)++;
  return cudaGetLastError();
}

cudaError_t launch_pre_moe(const float *x, uint32_t n_tokens, uint32_t D, const float *rms_weight, float eps, const float *shared_gate,
                           float *xn, float *shared_scale, cudaStream_t s, int *launches) {
  if (!rms_weight && !shared_gate) return cudaSuccess;
  const uintptr_t at = reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(rms_weight) | reinterpret_cast<uintptr_t>(shared_gate) | reinterpret_cast<uintptr_t>(xn);
  const cudaError_t e = launch_overlapped(D % 4 == 0 && at % 16 == 0 ? k_pre_moe<true> : k_pre_moe<false>, dim3(n_tokens), PRE_THREADS, 0, s, false, x, D,
                                          rms_weight, eps, shared_gate, xn, shared_scale);
  if (e != cudaSuccess) return e;
  if (launches) (*launches)++;
  return cudaGetLastError();
}

cudaError_t launch_dequant(int dtype, const uint8_t *src, float *dst, size_t n, cudaStream_t s) {
  int blocks = (int)((n + 255) / 256 < 148 * 16 ? (n + 255) / 256 : 148 * 16);
  if (blocks < 1) blocks = 1;
  if (dtype == MER_DTYPE_Q8_0)
    k_dequant<MER_DTYPE_Q8_0><<<blocks, 256, 0, s>>>(src, dst, n);
  else
    k_dequant<MER_DTYPE_Q4_0><<<blocks, 256, 0, s>>>(src, dst, n);
  return cudaGetLastError();
}

cudaError_t launch_dequant_packed(int dtype, const uint8_t *expert, int matrix, uint32_t D, uint32_t F, float *dst, cudaStream_t s) {
  if (dtype == MER_DTYPE_Q8_0)
    k_dequant_packed<MER_DTYPE_Q8_0><<<148 * 8, 256, 0, s>>>(expert, matrix, D, F, dst);
  else
    k_dequant_packed<MER_DTYPE_Q4_0><<<148 * 8, 256, 0, s>>>(expert, matrix, D, F, dst);
  return cudaGetLastError();
}

cudaError_t launch_repack(int dtype, const uint8_t *flat, uint8_t *packed, uint32_t D, uint32_t F, const SlotWrite &sw, cudaStream_t s) {
  if (dtype == MER_DTYPE_Q8_0)
    k_repack<MER_DTYPE_Q8_0><<<148 * 8, 256, 0, s>>>(flat, packed, D, F, sw);
  else
    k_repack<MER_DTYPE_Q4_0><<<148 * 8, 256, 0, s>>>(flat, packed, D, F, sw);
  return cudaGetLastError();
}
cudaError_t launch_slot_write(const SlotWrite &sw, cudaStream_t s) {
  k_slot_write<<<1, 1, 0, s>>>(sw);
  return cudaGetLastError();
}

cudaError_t launch_raw_matvec(int dtype, const uint8_t *w, const float *x, float *y, size_t rows, size_t cols, cudaStream_t s) {
  unsigned blocks = (unsigned)((rows + 7) / 8);
  if (dtype == MER_DTYPE_Q8_0)
    k_raw_matvec<MER_DTYPE_Q8_0><<<blocks, 256, 0, s>>>(w, x, y, rows, cols);
  else
    k_raw_matvec<MER_DTYPE_Q4_0><<<blocks, 256, 0, s>>>(w, x, y, rows, cols);
  return cudaGetLastError();
}

cudaError_t launch_host_in(const void *src, void *dst, size_t words, uint32_t *status, cudaStream_t s, int *launches) {
  const unsigned blocks = (unsigned)((words + 4 * HOST_COPY_THREADS - 1) / (4 * HOST_COPY_THREADS));
  k_host_in<<<blocks ? blocks : 1, HOST_COPY_THREADS, 0, s>>>(static_cast<const uint32_t *>(src), static_cast<uint32_t *>(dst), (uint32_t)words, status);
  if (launches) (*launches)++;
  return cudaGetLastError();
}
cudaError_t launch_host_out(const void *src, size_t stride, size_t rows, size_t words, void *dst, uint32_t *count, uint32_t *done, cudaStream_t s, int *launches) {
  if (launches) (*launches)++;
  return launch_overlapped(k_host_out, dim3(1), HOST_COPY_THREADS, 0, s, false, static_cast<const uint32_t *>(src), (uint32_t)stride, (uint32_t)rows,
                           (uint32_t)words, static_cast<uint32_t *>(dst), count, done);
}
cudaError_t launch_f16_to_f32(const uint16_t *src, float *dst, size_t n, cudaStream_t s) {
  k_f16_to_f32<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(src, dst, n);
  return cudaGetLastError();
}
cudaError_t launch_f32_to_f16(const float *src, uint16_t *dst, size_t n, cudaStream_t s) {
  k_f32_to_f16<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(src, dst, n);
  return cudaGetLastError();
}
