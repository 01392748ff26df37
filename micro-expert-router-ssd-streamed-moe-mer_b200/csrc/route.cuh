// Selection of one token's experts by one warp, shared by the router kernels.
#pragma once

#include <math_constants.h>
#include <stdint.h>

#include <climits>

#include "../../include/mer_b200.h"
#include "kernels.h"

namespace {

// Order of f32::total_cmp as a signed integer key (gating.rs:283-294 compares with total_cmp).
__device__ __forceinline__ int total_key(float f) {
  int b = __float_as_int(f);
  return b ^ (int)(((unsigned)(b >> 31)) >> 1);
}
__device__ __forceinline__ bool better(int ka, uint32_t ia, int kb, uint32_t ib) {
  return ka > kb || (ka == kb && ia < ib);
}

// Lane i < top_k gets the i-th pick; picks beyond n_sel (fewer finite scores than top_k) are MER_NONE with weight 0.
struct Pick {
  uint32_t id, n_sel;  // local expert index of this lane's pick; picks made (warp-uniform)
  float weight;
};

// Scoring, group filter, top-k and mixing weights of one token by one warp (LinearGate::route_with_scratch,
// gating.rs:395-476).  Scores and selection keys live in registers, EJ experts per lane (lane l holds experts l, l + 32,
// ...); s_score holds the logits on entry and the scores on return, s_sel is scratch for the group filter (E floats each).
// What bounds it is the latency of one warp's dependent steps, so every step is a handful of warp reductions: with the
// softmax sum added by one lane and the group scores by one lane per group, a token took 4.8 us on B200.
template <int EJ>
__device__ Pick route_token_reg(const RouterDev &r, float *s_score, float *s_sel, uint32_t *status) {
  const uint32_t E = r.num_experts, lane = threadIdx.x & 31, k = r.top_k;
  float sc[EJ];
#pragma unroll
  for (int j = 0; j < EJ; j++) {
    const uint32_t i = lane + 32 * j;
    sc[j] = i < E ? s_score[i] + (r.logit_bias ? __ldg(r.logit_bias + i) : 0.0f) : 0.0f;
  }
  if (r.scoring == MER_SCORE_SOFTMAX) {  // softmax_inplace (transformer.rs:2747-2819)
    float mx = -CUDART_INF_F;
    bool nan = false;
#pragma unroll
    for (int j = 0; j < EJ; j++)
      if (lane + 32 * j < E) mx = fmaxf(mx, sc[j]), nan |= sc[j] != sc[j];
    // the maximum of the total-order keys is the maximum of the values (-0 sorts below 0 and exponentiates alike)
    const int mk = __reduce_max_sync(0xffffffffu, total_key(mx));
    mx = __int_as_float(mk ^ (int)(((unsigned)(mk >> 31)) >> 1));
    nan = __any_sync(0xffffffffu, nan);
    if (nan || !isfinite(mx)) {
#pragma unroll
      for (int j = 0; j < EJ; j++) sc[j] = 1.0f / (float)E;
      if (lane == 0) atomicOr(status, MER_DEVSTAT_NONFINITE_ROUTER);
    } else {
      float sum = 0.0f;
#pragma unroll
      for (int j = 0; j < EJ; j++) {
        sc[j] = expf(sc[j] - mx);
        if (lane + 32 * j < E) sum += sc[j];
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
#pragma unroll
      for (int j = 0; j < EJ; j++) sc[j] = sc[j] / sum;  // sum >= 1: the largest term is exp(0)
    }
  } else {
#pragma unroll
    for (int j = 0; j < EJ; j++) sc[j] = 1.0f / (1.0f + expf(-sc[j]));
  }
  int keys[EJ];  // a taken or disallowed expert bids INT_MIN
  const uint32_t ng = r.n_group < 1 ? 1 : r.n_group;
  const bool grouped = ng > 1 && r.topk_group > 0 && r.topk_group < ng && (E % ng) == 0 && ng <= 64;
#pragma unroll
  for (int j = 0; j < EJ; j++) {
    const uint32_t i = lane + 32 * j;
    float sel = 0.0f;
    if (i < E) {
      s_score[i] = sc[j];
      sel = r.correction_bias ? sc[j] + __ldg(r.correction_bias + i) : sc[j];
      if (grouped) s_sel[i] = sel;
    }
    keys[j] = (i < E && isfinite(sel)) ? total_key(sel) : INT_MIN;
  }
  __syncwarp();
  if (grouped) {
    // group_filter_shape + select_top_groups (gating.rs:335-376): a group's score is the sum of its two best experts.
    // A power-of-two number of lanes shares each group; lane g of the first ng lanes (lane g - 32 for g >= 32) bids it.
    const uint32_t gs = E / ng, per = ng >= 32 ? 1u : 1u << (31 - __clz(32 / ng)), rounds = (ng * per + 31) / 32;
    uint64_t taken = 0;
    int gkey[2] = {INT_MIN, INT_MIN};
#pragma unroll 1
    for (uint32_t q = 0; q < rounds; q++) {
      const uint32_t g = q * 32 + lane / per;
      float top1 = -CUDART_INF_F, top2 = -CUDART_INF_F;
      if (g < ng) {
#pragma unroll 4
        for (uint32_t i = lane % per; i < gs; i += per) {
          const float v = s_sel[g * gs + i], s = v == v ? v : -CUDART_INF_F;
          top2 = fmaxf(top2, fminf(top1, s)), top1 = fmaxf(top1, s);
        }
      }
#pragma unroll 1
      for (uint32_t o = 1; o < per; o <<= 1) {
        const float b1 = __shfl_xor_sync(0xffffffffu, top1, o), b2 = __shfl_xor_sync(0xffffffffu, top2, o);
        top2 = fmaxf(fminf(top1, b1), fmaxf(top2, b2)), top1 = fmaxf(top1, b1);
      }
      const int key = total_key(top1 + (isfinite(top2) ? top2 : 0.0f));
      const int mine = __shfl_sync(0xffffffffu, key, (lane * per) & 31);
      if (q == 0 && lane < min(ng, 32u / per)) gkey[0] = mine;
      if (q == 1 && lane + 32 < ng) gkey[1] = mine;
    }
#pragma unroll 1
    for (uint32_t n = 0; n < r.topk_group; n++) {  // by (score desc, index asc)
      const int top = __reduce_max_sync(0xffffffffu, max(gkey[0], gkey[1]));
      const uint32_t id = __reduce_min_sync(0xffffffffu, gkey[0] == top ? lane : gkey[1] == top ? lane + 32 : MER_NONE);
      taken |= 1ull << (id & 63);
      if (lane == (id & 31)) {
        if (id < 32) gkey[0] = INT_MIN;
        else gkey[1] = INT_MIN;
      }
    }
    const uint32_t inv = (65536 + gs - 1) / gs;  // i / gs = i * inv >> 16 as i * gs < 65536
#pragma unroll
    for (int j = 0; j < EJ; j++) {
      const uint32_t i = lane + 32 * j;
      if (i < E && !(taken >> (i * inv >> 16) & 1)) keys[j] = INT_MIN;
    }
  }
  // top-k by (selection desc, id asc), non-finite skipped (gating.rs:315-333, 429-441).  Every lane sorts its own keys first
  // (neighbours change places while the later one is larger: equal keys keep their order), so that a pick is one warp maximum over the
  // lanes' first ones, a vote and a shift in the lane that wins.
  uint32_t ord[EJ];  // j of the key
#pragma unroll
  for (int j = 0; j < EJ; j++) ord[j] = j;
#pragma unroll
  for (int round = 0; round < EJ; round++) {
#pragma unroll
    for (int j = round & 1; j + 1 < EJ; j += 2) {
      const bool swap = keys[j + 1] > keys[j];
      const int ka = keys[j], kb = keys[j + 1];
      const uint32_t oa = ord[j], ob = ord[j + 1];
      keys[j] = swap ? kb : ka, keys[j + 1] = swap ? ka : kb, ord[j] = swap ? ob : oa, ord[j + 1] = swap ? oa : ob;
    }
  }
  uint32_t my_id = MER_NONE, n_sel = 0;
#pragma unroll 1
  for (uint32_t n = 0; n < k; n++) {
    const int top_key = __reduce_max_sync(0xffffffffu, keys[0]);
    if (top_key == INT_MIN) break;  // nothing left to pick
    const uint32_t tied = __ballot_sync(0xffffffffu, keys[0] == top_key);
    uint32_t top_lane = __ffs(tied) - 1;
    if (tied & (tied - 1))  // equal keys in several lanes: the lowest id wins
      top_lane = __reduce_min_sync(0xffffffffu, keys[0] == top_key ? lane + 32 * ord[0] : MER_NONE) & 31u;
    const uint32_t top_j = __shfl_sync(0xffffffffu, ord[0], top_lane);
    if (lane == top_lane) {
#pragma unroll
      for (int j = 0; j + 1 < EJ; j++) keys[j] = keys[j + 1], ord[j] = ord[j + 1];
      keys[EJ - 1] = INT_MIN;
    }
    if (lane == (n & 31)) my_id = top_lane + 32 * top_j;
    n_sel++;
  }
  // mixing weights = unbiased scores; renormalise; scale (gating.rs:443-474)
  float w = (lane < n_sel && my_id != MER_NONE) ? s_score[my_id] : 0.0f;
  if (r.normalise) {
    float sum = 0.0f;
    for (uint32_t i0 = 0; i0 < n_sel; i0 += 8) {  // slot order; the shuffles of eight slots are in flight together
      float v[8];
#pragma unroll
      for (int i = 0; i < 8; i++) v[i] = __shfl_sync(0xffffffffu, w, (i0 + i) & 31);
#pragma unroll
      for (int i = 0; i < 8; i++)
        if (i0 + i < n_sel) sum += v[i];
    }
    if (isfinite(sum) && sum > 0.0f) w = w / sum;
  }
  if (r.scaling != 1.0f && isfinite(r.scaling)) w = w * r.scaling;
  if (lane == 0 && n_sel < k) atomicOr(status, MER_DEVSTAT_SHORT_SELECTION);
  const bool have = lane < n_sel;
  return Pick{have ? my_id : MER_NONE, n_sel, have ? w : 0.0f};
}

// The same for any number of experts, from shared memory: s_ok is one byte per expert, s_groups / s_gscore 64 entries.
__device__ Pick route_token_any(const RouterDev &r, float *s_score, float *s_sel, uint8_t *s_ok, uint32_t *s_groups, float *s_gscore,
                                uint32_t *status) {
  const uint32_t E = r.num_experts, lane = threadIdx.x & 31;
  if (r.logit_bias)
#pragma unroll 1
    for (uint32_t i = lane; i < E; i += 32) s_score[i] += __ldg(r.logit_bias + i);
  __syncwarp();
  if (r.scoring == MER_SCORE_SOFTMAX) {
    // softmax_inplace (transformer.rs:2747-2819)
    float mx = -CUDART_INF_F;
    int nan = 0;
#pragma unroll 1
    for (uint32_t i = lane; i < E; i += 32) {
      float v = s_score[i];
      if (v != v)
        nan = 1;
      else if (v > mx)
        mx = v;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      nan |= __shfl_xor_sync(0xffffffffu, nan, o);
    }
    if (nan || !isfinite(mx)) {
#pragma unroll 1
      for (uint32_t i = lane; i < E; i += 32) s_score[i] = 1.0f / (float)E;
      if (lane == 0) atomicOr(status, MER_DEVSTAT_NONFINITE_ROUTER);
    } else {
#pragma unroll 1
      for (uint32_t i = lane; i < E; i += 32) s_score[i] = expf(s_score[i] - mx);
      __syncwarp();
      float sum = 0.0f;
      if (lane == 0) {  // the reference sums left to right; keep that order
        if ((E & 3u) == 0) {
          const float4 *s4 = reinterpret_cast<const float4 *>(s_score);  // E % 4 == 0 keeps every warp's array 16-byte aligned
#pragma unroll 4
          for (uint32_t i = 0; i < E / 4; i++) {
            const float4 v = s4[i];
            sum += v.x, sum += v.y, sum += v.z, sum += v.w;
          }
        } else {
#pragma unroll 1
          for (uint32_t i = 0; i < E; i++) sum += s_score[i];
        }
      }
      sum = __shfl_sync(0xffffffffu, sum, 0);
      if (sum > 0.0f)
#pragma unroll 1
        for (uint32_t i = lane; i < E; i += 32) s_score[i] = s_score[i] / sum;
    }
  } else {
#pragma unroll 1
    for (uint32_t i = lane; i < E; i += 32) s_score[i] = 1.0f / (1.0f + expf(-s_score[i]));
  }
  __syncwarp();
#pragma unroll 1
  for (uint32_t i = lane; i < E; i += 32) {
    s_sel[i] = r.correction_bias ? s_score[i] + r.correction_bias[i] : s_score[i];
    s_ok[i] = 1;
  }
  __syncwarp();
  // group_filter_shape + select_top_groups (gating.rs:335-376)
  const uint32_t ng = r.n_group < 1 ? 1 : r.n_group;
  const bool grouped = ng > 1 && r.topk_group > 0 && r.topk_group < ng && (E % ng) == 0 && ng <= 64;
  if (grouped) {
    const uint32_t gs = E / ng;
#pragma unroll 1
    for (uint32_t gi = lane; gi < ng; gi += 32) {
      float top1 = -CUDART_INF_F, top2 = -CUDART_INF_F;
#pragma unroll 1
      for (uint32_t i = 0; i < gs; i++) {
        float s = s_sel[gi * gs + i];
        if (s > top1) {
          top2 = top1;
          top1 = s;
        } else if (s > top2) {
          top2 = s;
        }
      }
      s_gscore[gi] = top1 + (isfinite(top2) ? top2 : 0.0f);
    }
    __syncwarp();
    if (lane == 0) {
      uint64_t taken = 0;
#pragma unroll 1
      for (uint32_t n = 0; n < r.topk_group; n++) {
        int bk = 0;
        uint32_t bi = MER_NONE;
#pragma unroll 1
        for (uint32_t g = 0; g < ng; g++) {
          if (taken >> g & 1) continue;
          int k = total_key(s_gscore[g]);
          if (bi == MER_NONE || better(k, g, bk, bi)) bk = k, bi = g;
        }
        taken |= 1ull << bi;
        s_groups[n] = bi;
      }
    }
    __syncwarp();
#pragma unroll 1
    for (uint32_t i = lane; i < E; i += 32) {
      bool ok = false;
#pragma unroll 1
      for (uint32_t n = 0; n < r.topk_group; n++) ok |= (s_groups[n] == i / gs);
      s_ok[i] = ok;
    }
    __syncwarp();
  }
  // top-k by (selection desc, id asc), non-finite skipped (gating.rs:315-333, 429-441)
  const uint32_t k = r.top_k;
  uint32_t my_id = MER_NONE;  // lane i keeps the i-th pick
  uint32_t n_sel = 0;
#pragma unroll 1
  for (uint32_t n = 0; n < k; n++) {
    int bk = 0;
    uint32_t bi = MER_NONE;
#pragma unroll 1
    for (uint32_t i = lane; i < E; i += 32) {
      float s = s_sel[i];
      if (!s_ok[i] || !isfinite(s)) continue;
      int key = total_key(s);
      if (bi == MER_NONE || key > bk) bk = key, bi = i;  // ascending scan keeps the lowest id on ties
    }
    // warp arg-max by (key desc, id asc): two warp reductions; lanes without a candidate bid the lowest key
    const int my_key = bi == MER_NONE ? INT_MIN : bk;
    const int top_key = __reduce_max_sync(0xffffffffu, my_key);
    const uint32_t top_id = __reduce_min_sync(0xffffffffu, (bi != MER_NONE && my_key == top_key) ? bi : MER_NONE);
    bk = top_key, bi = top_id;
    if (bi == MER_NONE) break;
    if (lane == 0) s_ok[bi] = 0;
    if (lane == (n & 31)) my_id = bi;
    n_sel++;
    __syncwarp();
  }
  // mixing weights = unbiased scores; renormalise; scale (gating.rs:443-474)
  float w = (lane < n_sel && my_id != MER_NONE) ? s_score[my_id] : 0.0f;
  if (r.normalise) {
    float sum = 0.0f;
#pragma unroll 1
    for (uint32_t i = 0; i < n_sel; i++) sum += __shfl_sync(0xffffffffu, w, i);  // slot order
    if (isfinite(sum) && sum > 0.0f) w = w / sum;
  }
  if (r.scaling != 1.0f && isfinite(r.scaling)) w = w * r.scaling;
  if (lane == 0 && n_sel < k) atomicOr(status, MER_DEVSTAT_SHORT_SELECTION);
  const bool have = lane < n_sel;
  return Pick{have ? my_id : MER_NONE, n_sel, have ? w : 0.0f};
}

// E floats of logits (scores on return) and E of scratch; beyond 256 experts also s_ok, s_groups and s_gscore.
__device__ __forceinline__ Pick route_token(const RouterDev &r, float *s_score, float *s_sel, uint8_t *s_ok, uint32_t *s_groups, float *s_gscore,
                                            uint32_t *status) {
  if (r.num_experts <= 128) return route_token_reg<4>(r, s_score, s_sel, status);
  if (r.num_experts <= 256) return route_token_reg<8>(r, s_score, s_sel, status);
  return route_token_any(r, s_score, s_sel, s_ok, s_groups, s_gscore, status);
}

}  // namespace
