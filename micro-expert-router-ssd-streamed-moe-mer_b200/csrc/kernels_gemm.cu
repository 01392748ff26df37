// Grouped expert FFN for token groups of a dozen tokens and more (prefill, expert-parallel decode):
// tcgen05 tensor-core GEMM per (expert, 256 weight rows, up to 128 or 256 tokens) on pairs of CTAs, accumulators in TMEM.
//
//   D[256 weight rows x N tokens] += A[256 x 32] * B[N x 32]^T      per 32-value block of K
//
//   * Two CTAs (a cluster, cta_group::2) multiply 128 weight rows each against one B operand of which each holds half of the
//     token rows: half the activation traffic and half the MMA instructions per weight row of single CTAs.
//   * A never touches shared memory as an operand: the packed Q4_0 / Q8_0 tile chunks of layout.cuh
//     are streamed global -> shared by bulk async copies, sixteen warps dequantise them block by block into
//     two f16 operands, hi = f16(d*q) and lo = d*q - hi (exact: an 11-bit scale times an 8-bit integer
//     has at most 19 significant bits), and store them straight into TENSOR MEMORY (tcgen05.st; a thread
//     owns one weight row), from where the MMA reads its A operand.  Eight A stages live in TMEM beside
//     the two accumulators; a block is converted before its stage is waited for.
//   * B is the activation rows as f16 hi + lo parts (22 significant bits after an exact power-of-two
//     per-row scaling), written once in group order by k_split_rows, so that a pass is a run of rows and one tiled copy
//     fetches 64 values of all of them (128-byte swizzle; a tensor map per pass width).
//   * Three products per 16 values of K (hi*hi, hi*lo, lo*hi; lo*lo is below fp32 resolution) accumulate
//     in fp32 in TMEM, so the result matches the fp32 reference to ~1e-4 of the output RMS instead of f16's 2e-3.
//   * Warp roles: 0 = producer of the activation stages, 1 = MMA issuer (of the pair's first CTA; one elected lane issues
//     predicated instructions; every operand is computed in uniform registers) and TMEM owner, 2..9 = epilogue (two groups
//     of four, one per accumulator buffer), 10..25 = dequantisers (two teams of two per quarter of the rows, two blocks of every second
//     weight stage each), 26 and 27 = producers of the weight stages (lanes 0..3 copy one packed tile each).
// What bounds it: the way of A through tensor memory on passes of up to 64 tokens, the MMAs from about 80 on, the power limit on full-width
// ones.  A group of four blocks takes 1050 cycles on a pass of 32 tokens (1750 before) and 1150 on one of 80; the MMAs of N columns N / 2 each,
// 24 a group, so 380 and 960 (alone, with A in tensor memory, they run at that rate for every N, whatever else uses tensor or shared memory).  The
// rest is the cycle MMAs -> done -> store -> arrival at the issuer of the other CTA, 2000 cycles of which two are in flight.
// Us a pass, L2 flushed, without uniform operands, one activation copy a group, two weight producers and two teams of dequantisers / now, one box: 256 tokens on 8
// experts of 4096 x 14336 689 / 624, 2 layers of 2048 on 128 of 2048 x 768 1284 / 1214; 4096 on 256 of 7168 x 2048, at the power limit, 8565 / 8524: even.
// Tried without gain: one MMA for hi * [hi | lo] of passes up to 32 tokens, the conversion of both blocks ahead of the wait (spills: 531 / 522),
// commits or groups of two blocks, fewer instructions in the conversion, a look at the issuer's next barrier ahead.
// Every wait is bounded; on expiry the CTA latches MER_DEVSTAT_TIMEOUT, stops issuing work, waits
// (bounded) for its copies and MMAs in flight, frees its TMEM and returns.
#include <cuda.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

#include "../../include/mer_b200.h"
#include "act_rows.h"
#include "decode.cuh"
#include "kernels.h"
#include "layout.cuh"
#include "ptx.cuh"

namespace {

constexpr int G_WARPS = 28, G_THREADS = G_WARPS * 32;
constexpr int W_PRODUCER = 0, W_MMA = 1, W_EPI0 = 2, W_DQ0 = 10, W_WEIGHTS = 26, WEIGHT_WARPS = 2;
constexpr int EPI_WARPS = 4, DQ_WARPS = 16;  // EPI_WARPS per accumulator
constexpr uint32_t PAIR = 2;             // CTAs of a cluster: they share the B operand, each holding half of its rows
constexpr uint32_t RAW_BLOCKS = 4;       // blocks of K per weight stage (per packed tile: one bulk copy)
constexpr uint32_t G_HEADER = 5120;      // mbarriers, TMEM base, and from byte 1024 the epilogue groups' per-pass tables (2 KB each)
constexpr uint32_t TMEM_COLS = 512;      // [0, 256): two accumulator buffers of up to 128 columns; [256, 512): A stages
constexpr uint32_t TMEM_A0 = 256, A_STAGES = 8, A_STAGE_COLS = 32;  // a stage = one block: 16 columns hi + 16 columns lo
constexpr uint32_t RAW_STAGES = 4;
// The MMA issuer synchronises with its producers once per GROUP blocks of K: it waits for the group's activation stage (b_full: the bytes of both
// CTAs' copies) and for its A stages of both CTAs (a_full: the dequantiser warps of the pair that convert it), issues the group's
// MMAs and commits done[] in both CTAs, which releases all of it.  The barriers are counted by groups, of which no more than n_b are in flight.
constexpr uint32_t GROUP = 4, A_RING = A_STAGES / GROUP, DONE_RING = 16, FULL_RING = 8;
constexpr uint32_t CHUNKS = GROUP * 32 / ACT_CHUNK_K;
constexpr uint32_t PASS_TOKENS = 256;    // tokens of a pass at most: N of one MMA
// A pass of up to BUF_TOKENS takes one of the two accumulator buffers and one activation stage a group; a wider one takes both buffers (its MMAs then
// wait for the epilogue of the item before) and two stages: what it saves is a second conversion of the weights.
constexpr uint32_t BUF_TOKENS = 128;
constexpr uint32_t B_STAGE = CHUNKS * 2 * (BUF_TOKENS / PAIR) * 128;  // of each chunk the hi rows, then the lo rows
static_assert(RAW_BLOCKS == GROUP && DQ_WARPS == 4 * RAW_BLOCKS && A_RING == 2, "a weight stage is a group; two of its blocks for each of a quarter's warps of a team");
constexpr float POW2_SCALE_TARGET = 9;   // activations are scaled so that the row maximum lies in [256, 512)

struct GemmParams {
  MoeDispatch d;
  int phase;               // 0 = gate/up (+SiLU*mul), 1 = down
  const float *unscale;    // 1 / scale of each activation row
  uint32_t rows;           // F (gate/up) or D (down)
  uint32_t kb_total;       // 32-value blocks per weight row
  uint32_t n_b;            // stages of the activation ring
  float *out;              // phase 0: h [P x F]; phase 1: y [P x D]
};

// The activation matrix in boxes of 8, 16 .. 128 rows (half a pass's width) x both parts x a group's chunks of 64 values.
struct ActMaps {
  CUtensorMap m[PASS_TOKENS / 16];
};

// ------------------------------------------------------------------------------ tcgen05 PTX
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// One lane of a converged warp.  The MMA warp runs its loops and waits with all 32 lanes, so that every address and
// descriptor it computes is warp-uniform; the lane elected ONCE at the start issues the tcgen05.mma / tcgen05.commit
// instructions, as predicated instructions (no branch around them).  Measured on the way here: the whole loop inside
// `if (lane == 0)` cost ~85 cycles of issue time per MMA, an elect.sync + branch around every single MMA ~65, either
// of them more than a narrow MMA takes to execute.
__device__ __forceinline__ uint32_t elect_one() {
  uint32_t pred;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(pred));
  return pred;
}
__device__ __forceinline__ void tc_commit(uint32_t leader, uint64_t *bar) {
  asm volatile(
      "{\n .reg .pred q;\n setp.ne.b32 q, %1, 0;\n"
      " @q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %2;\n}\n" ::"r"(smem_u32(bar)),
      "r"(leader), "h"((uint16_t)3)
      : "memory");
}
// K-major rows of 128 bytes, swizzled in atoms of 8 rows (1024 bytes).  Bits: start >> 4 [0,14), LBO (not used) [16,30),
// SBO = 1024 >> 4 between atoms [32,46), version 1 [46,48), 128-byte swizzle = 2 [61,64).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
// f16 x f16 -> f32, both operands K-major, M = 256 (128 rows in each CTA of the pair), N = n.
__host__ __device__ constexpr uint32_t instr_desc(uint32_t n) { return (1u << 4) | ((n >> 3) << 17) | ((256u >> 4) << 24); }
// The same shared-memory address in the pair's first CTA, which issues the MMAs and holds the barriers it waits on.
__device__ __forceinline__ uint32_t leader_addr(const void *p) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(smem_u32(p)));
  return a;
}
// The box of `map` at row r and chunk `chunk` of the activation matrix into this CTA's shared memory (128-byte rows, swizzled: the rows' hi parts
// of the first chunk, their lo parts, the same of the second); the bytes are counted on a barrier of the pair's first CTA.
__device__ __forceinline__ void group_g2s(uint32_t dst, const CUtensorMap *map, uint32_t r, uint32_t chunk, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3, %2, %4}], [%5];" ::"r"(dst),
      "l"(map), "r"(0), "r"(r), "r"(chunk), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// A operand read from tensor memory (lane = row, a 32-bit column = two consecutive values of K), B through a descriptor.
// Called by the whole (converged) warp; only the lane with leader != 0 issues.
__device__ __forceinline__ void tc_mma_ts(uint32_t leader, uint32_t d_tmem, uint32_t a_tmem, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.b32 q, %5, 0;\n setp.ne.b32 p, %4, 0;\n"
      " @q tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b), "r"(idesc), "r"(accumulate), "r"(leader)
      : "memory");
}
__device__ __forceinline__ void tc_mma_ts_acc(uint32_t leader, uint32_t d_tmem, uint32_t a_tmem, uint64_t b, uint32_t idesc) {
  tc_mma_ts(leader, d_tmem, a_tmem, b, idesc, 1u);
}
// 32 columns of this thread's TMEM lane (lane = 32 * (warp % 4) + lane id).
__device__ __forceinline__ void tc_st32(uint32_t taddr, const uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};\n" ::"r"(taddr),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]),
      "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]),
      "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]),
      "r"(v[31])
      : "memory");
}
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// 16 columns of this thread's TMEM lane.
__device__ __forceinline__ void tc_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
      "tcgen05.wait::ld.sync.aligned;\n"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
        "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ __half2 bits_h2(uint32_t v) { return *reinterpret_cast<__half2 *>(&v); }

// Token columns of a pass: its count rounded up to 16.
__host__ __device__ constexpr uint32_t pass_width(uint32_t count) { return (count + 15u) & ~15u; }
// A group of at most SPLIT_TOKENS tokens (always a single pass) leaves half of its accumulator buffer free: the two small
// products go there and are added at the end, so that the large one is rounded by its own additions only.  The
// rule looks at the group, not at the pass, so that the order of a token's additions depends only on how many tokens its
// expert received, never on which pass it landed in: results stay bit-identical from run to run although large
// dispatches are grouped with atomics.
constexpr uint32_t SPLIT_TOKENS = BUF_TOKENS / 2;

struct Ring {
  uint32_t stage = 0, round = 0, n;
  __device__ explicit Ring(uint32_t n_) : n(n_) {}
  __device__ void advance() {
    if (++stage == n) stage = 0, round++;
  }
};

// The ring of activation stages (an even number of at most eight) as its producer and the issuer count it: a group of blocks takes one stage, or
// two adjacent ones from an even one on.
struct StageRing {
  uint32_t n, at = 0;
  __device__ explicit StageRing(uint32_t n_) : n(n_) {}
  __device__ __forceinline__ uint32_t take(bool wide) {
    if (wide) at = (at + 1) & ~1u;
    if (at >= n) at = 0;
    const uint32_t st = at;
    at += wide ? 2 : 1;
    return st;
  }
};

template <int DT>
__global__ void __cluster_dims__(PAIR, 1, 1) __launch_bounds__(G_THREADS, 1) k_ffn_gemm(const GemmParams p, const __grid_constant__ ActMaps maps) {
  extern __shared__ __align__(1024) uint8_t smem[];
  constexpr uint32_t BB = DT == MER_DTYPE_Q4_0 ? MER_Q4_BLOCK_BYTES : MER_Q8_BLOCK_BYTES;
  constexpr uint32_t TILE_RAW = RAW_BLOCKS * 16 * BB;  // bytes of RAW_BLOCKS blocks of one packed tile (1152 / 2176)
  constexpr uint32_t RAW_BYTES = 8 * TILE_RAW;
  const MoeDispatch &d = p.d;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  const uint32_t rank = blockIdx.x & 1;
  const uint32_t m_tiles = p.rows / (p.phase == 0 ? 64u : 128u);  // 128-row MMA tiles (8 packed tiles each)
  const uint32_t m_pairs = (m_tiles + 1) / 2;                     // the second CTA of an odd last pair repeats the last tile, unwritten
  const uint32_t n_groups = p.kb_total / GROUP;
  const uint32_t n_passes = *d.n_passes;
  // Items (pass, 256 rows) are dealt round-robin: the pairs running at any moment work on a dozen
  // neighbouring passes, so the activation rows they all re-read stay in L2.
  const uint32_t n_items = n_passes * m_pairs;
  const uint32_t item_beg = blockIdx.x / PAIR, item_step = gridDim.x / PAIR;
  if (item_beg >= n_items) return;

  uint64_t *bars = reinterpret_cast<uint64_t *>(smem);
  uint64_t *raw_full = bars, *raw_empty = bars + 8, *a_full = bars + 16, *b_full = bars + 24, *done = bars + 32,
           *acc_full = bars + 48, *acc_empty = bars + 50, *drain = bars + 52;
  uint32_t *s_tmem = reinterpret_cast<uint32_t *>(smem + 512);
  volatile uint32_t *s_abort = reinterpret_cast<volatile uint32_t *>(smem + 516);
  uint8_t *s_b = smem + G_HEADER;
  uint8_t *s_raw = s_b + p.n_b * B_STAGE;

  if (threadIdx.x == 0) {
    // filled by the weight producers, left by a team of dequantisers
    for (uint32_t s = 0; s < RAW_STAGES; s++) mbar_init(&raw_full[s], WEIGHT_WARPS), mbar_init(&raw_empty[s], DQ_WARPS / 2);
    for (uint32_t s = 0; s < FULL_RING; s++) mbar_init(&a_full[s], PAIR * DQ_WARPS / 2), mbar_init(&b_full[s], 1);
    for (uint32_t s = 0; s < DONE_RING; s++) mbar_init(&done[s], 1);
    for (uint32_t s = 0; s < 2; s++) mbar_init(&acc_full[s], 1), mbar_init(&acc_empty[s], PAIR * EPI_WARPS);
    mbar_init(drain, 1);
    *s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == W_MMA) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(s_tmem)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  cluster_sync();
  tc_fence_after();
  // The CTA owns all 512 columns of its SM's tensor memory, so the allocation starts at lane 0, column 0.  Using the
  // constant instead of the value read back lets every TMEM address below be computed in uniform registers: with the
  // loaded value each MMA took ~57 cycles to issue, with the constant ~35.  Should the allocator ever answer otherwise,
  // the kernel gives the columns back, latches the error status and leaves.
  constexpr uint32_t tmem_base = 0;
  if (*s_tmem != tmem_base) {
    if (warp == W_MMA) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(*s_tmem), "r"(TMEM_COLS) : "memory");
    if (threadIdx.x == 0) atomicOr(p.d.status, MER_DEVSTAT_TIMEOUT);
    return;
  }

  const size_t proj_bytes = (size_t)d.D * d.F / 32 * BB;
  const size_t tile_bytes = (size_t)p.kb_total * 16 * BB;
  const size_t region = p.phase == 0 ? 0 : 2 * proj_bytes;
  // What a role needs to know of its items, fetched for 32 of them at a time, one per lane: the three dependent loads
  // behind an expert's address would otherwise stall every role at the start of every item.
  struct Items {
    uint64_t base = 0;
    uint32_t start = 0, count = 0, split = 0;
    __device__ void fetch(const MoeDispatch &d, uint32_t item, uint32_t n_items, uint32_t m_pairs) {
      if (item >= n_items) return;
      const uint32_t pass = item / m_pairs, g = __ldg(d.pass_group + pass), eid = d.group_expert[g];
      split = __ldg(d.offsets + g + 1) - __ldg(d.offsets + g) <= SPLIT_TOKENS;
      start = __ldg(d.pass_start + pass), count = __ldg(d.pass_count + pass);
      base = eid < d.max_experts ? reinterpret_cast<uint64_t>(d.expert_ptr[eid]) : 0;
    }
  } items;
  uint32_t item_no = 0;  // running number of the role's item
  auto next_item = [&](uint32_t item, uint32_t &start, uint32_t &count, bool *split = nullptr) -> const uint8_t * {
    const uint32_t k = item_no++ & 31;
    if (k == 0) items.fetch(d, item + lane * item_step, n_items, m_pairs);
    start = __shfl_sync(0xffffffffu, items.start, k), count = __shfl_sync(0xffffffffu, items.count, k);
    if (split) *split = __shfl_sync(0xffffffffu, items.split, k) != 0;
    return reinterpret_cast<const uint8_t *>(__shfl_sync(0xffffffffu, items.base, k));
  };
  uint32_t pstart, pcount;
  bool split;
  bool ok = true;

  if (warp == W_PRODUCER) {
    // ------------------------------------------------------------------------ producer of the activation stages
    // one stage = one group of blocks of K of this CTA's half of the pass's rows: one copy.  Four of 64 values and a part each kept this warp busy for
    // 1000 cycles a group.  A stage is free again when the MMAs of the group that used it have run: the issuer's done[] commit says so.
    StageRing rb(p.n_b);
    uint32_t holder = 0;  // lane i: 1 + the group that took stage i last
    uint32_t pg = 0;  // groups issued so far, over all items (the issuer counts the same way)
    for (uint32_t item = item_beg; item < n_items && ok; item += item_step) {
      if (!next_item(item, pstart, pcount)) continue;
      const uint32_t width = pass_width(pcount), row = pstart + rank * (width / PAIR);
      const CUtensorMap *map = &maps.m[width / 16 - 1];
      const bool wide = width > BUF_TOKENS;
      for (uint32_t gi = 0; gi < n_groups && ok; gi++, pg++) {
        const uint32_t stage = rb.take(wide);
        uint64_t *bar = &b_full[pg % FULL_RING];
        // 1 + the newest group that has had one of these stages
        const bool mine = lane == stage || (wide && lane == stage + 1);
        const uint32_t busy = __reduce_max_sync(0xffffffffu, mine ? holder : 0u);
        if (mine) holder = pg + 1;
        if (busy) ok = mbar_wait_cluster(&done[(busy - 1) % DONE_RING], ((busy - 1) / DONE_RING) & 1);
        if (*s_abort) ok = false;
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        if (lane == 0) {
          if (rank == 0) mbar_expect_tx(bar, CHUNKS * width * 2 * 128);  // both CTAs' bytes
          group_g2s(smem_u32(s_b) + stage * B_STAGE, map, row, gi * CHUNKS, leader_addr(bar));
        }
      }
    }
    if (!ok) {
      if (lane == 0) *s_abort = 1, atomicOr(d.status, MER_DEVSTAT_TIMEOUT);
      // copies already in flight get a bounded chance to land before the pair's shared memory is released
      if (rank == 0)
        for (uint32_t s = 0; s < FULL_RING; s++) mbar_drain(&b_full[s], 0, 10000000ull), mbar_drain(&b_full[s], 1, 10000000ull);
    }
  } else if (warp == W_MMA) {
    // -------------------------------------------------------------------------- MMA issuer (of the pair: its first CTA)
    if (rank == 0) {
    // The whole warp walks the loops and waits (every value it computes is warp-uniform); the elected lane issues.
    // one step = one 32-value block of K: two instructions of 16 values for each of the three operand pairings
    StageRing rb(p.n_b);
    const uint32_t leader = elect_one();  // the warp is converged here; the same lane issues from now on
    uint32_t next_buf = 0, uses0 = 0, uses1 = 0;  // accumulator buffer of the next item that takes one; items that have used either
    uint32_t grp = 0;     // groups of GROUP blocks issued so far, over all items; A-stage half = grp & 1
    // B descriptors differ only in their start-address field: one base, then 64-bit adds of (byte offset >> 4).
    // (The ring lies well inside the 256 KB the 14-bit field spans, so the adds never carry out of it.)
    const uint64_t b_desc0 = smem_desc(smem_u32(s_b));
    // One item's K loop for a pass of WIDTH columns.  WIDTH is a template argument because everything the MMA instruction
    // takes (descriptors, TMEM addresses) must sit in uniform registers: values derived from kernel parameters and
    // constants are computed there directly, values derived from a loaded pass count had to be moved over per
    // instruction (measured: +25 % issue time).
    auto run_item = [&](auto width_tag, auto split_tag) {
      constexpr uint32_t WIDTH = decltype(width_tag)::value;
      constexpr uint32_t LO = decltype(split_tag)::value ? SPLIT_TOKENS : 0;  // columns of the small products
      constexpr uint32_t idesc = instr_desc(WIDTH);
      constexpr bool WIDE = WIDTH > BUF_TOKENS;
      constexpr uint32_t PART = WIDTH / PAIR * 128;  // bytes of the hi or the lo rows of a chunk
      const uint32_t buf = WIDE ? 0 : next_buf;
      // the previous item of the buffer (of both) has been drained
      if ((WIDE || buf == 0) && uses0 > 0) ok = mbar_wait_tmem(&acc_empty[0], (uses0 - 1) & 1);
      if ((WIDE || buf == 1) && uses1 > 0) ok = mbar_wait_tmem(&acc_empty[1], (uses1 - 1) & 1) && ok;
      ok = __all_sync(0xffffffffu, ok);  // warp-uniform by construction; the votes also tell the compiler so
      uint32_t acc = 0;  // the item's first MMA overwrites the accumulator
      for (uint32_t left = n_groups; left > 0 && ok; left--) {
        // A reduction's result sits in a uniform register, and so does all that is computed from it.  Values that the loop over the items carries had to be
        // moved over for every instruction: 34 cycles to issue one instead of 14.
        const uint32_t at = __reduce_max_sync(0xffffffffu, rb.take(WIDE) << 2 | (grp % A_RING) << 1 | buf);
        const uint32_t stage = at >> 2, a_grp = tmem_base + TMEM_A0 + (at >> 1 & 1) * GROUP * A_STAGE_COLS, d_tmem = tmem_base + (at & 1) * 128;
        // (the activations land well ahead of the A stages: their wait, 200 cycles of which are its acquire at cluster scope, costs nothing)
        ok = mbar_wait_cluster(&b_full[grp % FULL_RING], (grp / FULL_RING) & 1);
        if (ok) ok = mbar_wait_tmem(&a_full[grp % FULL_RING], (grp / FULL_RING) & 1);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        const uint64_t b_stage = b_desc0 + (uint64_t)(stage * (B_STAGE >> 4));
        uint64_t *freed = &done[grp % DONE_RING];
        grp++;
#pragma unroll
        for (uint32_t b4 = 0; b4 < GROUP; b4++) {
          const uint32_t a_hi = a_grp + b4 * A_STAGE_COLS, a_lo = a_hi + 16;
          const uint64_t b_blk = b_stage + (uint64_t)(((b4 >> 1) * 2 * PART + (b4 & 1) * 64) >> 4);
#pragma unroll
          for (uint32_t j = 0; j < 2; j++) {  // 16 values of K per instruction: 8 TMEM columns of A, 32 bytes of a row of B
            const uint64_t dbh = b_blk + (uint64_t)(j * 2), dbl = dbh + (PART >> 4);
            if (b4 > 0 || j > 0) acc = 1;
            tc_mma_ts(leader, d_tmem, a_hi + j * 8, dbh, idesc, acc);
            tc_mma_ts(leader, d_tmem + LO, a_hi + j * 8, dbl, idesc, LO ? acc : 1u);
            tc_mma_ts_acc(leader, d_tmem + LO, a_lo + j * 8, dbh, idesc);
          }
        }
        tc_commit(leader, freed);  // frees the group's A stages and its activation stage, in both CTAs
      }
      if (ok) {
        tc_commit(leader, &acc_full[buf]);
        if (WIDE) tc_commit(leader, &acc_full[1]);
      }
      if (WIDE || buf == 0) uses0++;
      if (WIDE || buf == 1) uses1++;
      next_buf = WIDE ? 0 : buf ^ 1;
    };
    for (uint32_t item = item_beg; item < n_items && ok; item += item_step) {
      if (!next_item(item, pstart, pcount, &split)) continue;
      // the MMA is as wide as the pass has tokens (rounded up to 16 columns)
      using T = std::true_type;
      using F = std::false_type;
      const uint32_t w16 = pass_width(pcount) >> 4;
      if (split) {
        switch (w16) {
          case 1: run_item(std::integral_constant<uint32_t, 16>{}, T{}); break;
          case 2: run_item(std::integral_constant<uint32_t, 32>{}, T{}); break;
          case 3: run_item(std::integral_constant<uint32_t, 48>{}, T{}); break;
          default: run_item(std::integral_constant<uint32_t, 64>{}, T{}); break;
        }
      } else {
        switch (w16) {
          case 1: run_item(std::integral_constant<uint32_t, 16>{}, F{}); break;
          case 2: run_item(std::integral_constant<uint32_t, 32>{}, F{}); break;
          case 3: run_item(std::integral_constant<uint32_t, 48>{}, F{}); break;
          case 4: run_item(std::integral_constant<uint32_t, 64>{}, F{}); break;
          case 5: run_item(std::integral_constant<uint32_t, 80>{}, F{}); break;
          case 6: run_item(std::integral_constant<uint32_t, 96>{}, F{}); break;
          case 7: run_item(std::integral_constant<uint32_t, 112>{}, F{}); break;
          case 8: run_item(std::integral_constant<uint32_t, 128>{}, F{}); break;
          case 9: run_item(std::integral_constant<uint32_t, 144>{}, F{}); break;
          case 10: run_item(std::integral_constant<uint32_t, 160>{}, F{}); break;
          case 11: run_item(std::integral_constant<uint32_t, 176>{}, F{}); break;
          case 12: run_item(std::integral_constant<uint32_t, 192>{}, F{}); break;
          case 13: run_item(std::integral_constant<uint32_t, 208>{}, F{}); break;
          case 14: run_item(std::integral_constant<uint32_t, 224>{}, F{}); break;
          case 15: run_item(std::integral_constant<uint32_t, 240>{}, F{}); break;
          default: run_item(std::integral_constant<uint32_t, 256>{}, F{}); break;
        }
      }
    }
    if (!ok && lane == 0) *s_abort = 1, atomicOr(d.status, MER_DEVSTAT_TIMEOUT);
    __syncwarp();
    // nothing may still be writing TMEM when it is freed
    tc_commit(leader, drain);
    (void)mbar_wait(drain, 0);
    __syncwarp();
    }
  } else if (warp >= W_WEIGHTS) {
    // ------------------------------------------------------------------------ producers of the weight stages
    // one stage = RAW_BLOCKS blocks of K of the item's eight packed tiles; each of two warps copies the chunks of four, a lane one (a copy takes the
    // warp some 110 cycles; eight of them, 900 a group, were more than what the MMAs of a narrow pass take)
    constexpr uint32_t TILES = 8 / WEIGHT_WARPS;
    const uint32_t tile = (warp - W_WEIGHTS) * TILES + lane % TILES;
    Ring raw(RAW_STAGES);
    for (uint32_t item = item_beg; item < n_items && ok; item += item_step) {
      const uint8_t *base = next_item(item, pstart, pcount);
      if (!base) continue;
      const uint32_t mt = min((item % m_pairs) * PAIR + rank, m_tiles - 1);
      const uint8_t *src = base + region + (size_t)(mt * 8 + tile) * tile_bytes;
      for (uint32_t gi = 0; gi < p.kb_total / RAW_BLOCKS && ok; gi++) {
        if (raw.round > 0) ok = mbar_wait(&raw_empty[raw.stage], (raw.round - 1) & 1);  // every dequantiser warp has left the stage
        if (*s_abort) ok = false;
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        if (lane == 0) mbar_expect_tx(&raw_full[raw.stage], RAW_BYTES / WEIGHT_WARPS);
        __syncwarp();
        if (lane < TILES) bulk_g2s(s_raw + raw.stage * RAW_BYTES + tile * TILE_RAW, src + (size_t)gi * TILE_RAW, TILE_RAW, &raw_full[raw.stage]);
        raw.advance();
      }
    }
    if (!ok) {
      if (lane == 0) *s_abort = 1, atomicOr(d.status, MER_DEVSTAT_TIMEOUT);
      // weight copies already in flight get a bounded chance to land before the CTA's shared memory is released
      for (uint32_t s = 0; s < RAW_STAGES; s++) (void)mbar_wait(&raw_full[s], 0), (void)mbar_wait(&raw_full[s], 1);
    }
  } else if (warp >= W_DQ0) {
    // ------------------------------------------------------------------------ dequantisers
    // A thread owns one weight row of the item: TMEM lane 32 * (warp % 4) + lane, i.e. packed tile 2q + lane / 16,
    // row slot lane % 16.  Per block it reads the row's 32 quants from the tile chunk in shared memory and stores
    // 16 columns of hi and 16 of lo.  Two teams of eight warps take the groups in turn, a warp two adjacent blocks of each of its
    // team's: one team converts while the other waits and stores (256 tokens on 8 experts of 4096 x 14336 535 us, with a block of every group a warp 569).
    const uint32_t q = warp & 3, team = (warp - W_DQ0) >> 2 & 1, mine = (warp - W_DQ0) >> 3 << 1;  // quarter of the rows; first of the two blocks
    const uint32_t T = 2 * q + (lane >> 4), g = lane & 7, half = (lane >> 3) & 1;
    const __half2 zp = DT == MER_DTYPE_Q4_0 ? __floats2half2_rn(1032.0f, 1032.0f) : __floats2half2_rn(1152.0f, 1152.0f);
    constexpr bool EARLY = DT == MER_DTYPE_Q4_0;  // the second block's integers ahead of the wait
    constexpr int RAW_WORDS = DT == MER_DTYPE_Q4_0 ? 4 : 8;
    uint32_t groups = 0;  // groups of blocks before this item
    bool ready = false;   // the weight stage has been seen full
    const uint32_t tile0 = smem_u32(s_raw) + T * TILE_RAW;
    const uint32_t a_tmem = tmem_base + ((q * 32u) << 16) + TMEM_A0 + mine * A_STAGE_COLS;
    // the quants of this thread's row in block `blk` of a stage, and their scale
    auto load = [&](uint32_t src, uint32_t blk, uint32_t (&w)[RAW_WORDS], uint32_t &scale) {
      if (DT == MER_DTYPE_Q8_0) {
        src += blk * 544;
        scale = lds32(src + 512 + g * 4);
#pragma unroll
        for (int t = 0; t < 4; t++) {  // values 8t .. 8t+7
          const uint2 v = lds64(src + packed_piece(g, t) * 16 + half * 8);
          w[2 * t] = v.x, w[RAW_WORDS > 4 ? 2 * t + 1 : 0] = v.y;
        }
      } else {
        // block-pair record: 16 bytes per (g, t) = words (slot g, blk 0), (slot g+8, blk 0), (slot g, blk 1), (slot g+8, blk 1);
        // byte i of a word holds values 4t+i (low nibble) and 16+4t+i (high nibble) of its block
        src += (blk >> 1) * 576;
        scale = lds32(src + 512 + g * 8 + (blk & 1) * 4);
#pragma unroll
        for (int t = 0; t < 4; t++) w[t] = lds32(src + packed_piece(g, t) * 16 + ((blk & 1) * 2 + half) * 4);
      }
    };
    // The quants as f16 pairs, exact: column c holds values (2c, 2c+1) of the block.
    auto integers = [&](const uint32_t (&w)[RAW_WORDS], __half2 (&q)[16]) {
#pragma unroll
      for (int t = 0; t < 4; t++) {
        if (DT == MER_DTYPE_Q8_0) {
          const uint32_t a = w[2 * t], b = w[RAW_WORDS > 4 ? 2 * t + 1 : 0];
          q[4 * t + 0] = __hsub2(bits_h2(__byte_perm(a, 0x64646464u, 0x4140)), zp), q[4 * t + 1] = __hsub2(bits_h2(__byte_perm(a, 0x64646464u, 0x4342)), zp);
          q[4 * t + 2] = __hsub2(bits_h2(__byte_perm(b, 0x64646464u, 0x4140)), zp), q[4 * t + 3] = __hsub2(bits_h2(__byte_perm(b, 0x64646464u, 0x4342)), zp);
        } else {
          const uint32_t lows = w[t] & 0x0F0F0F0Fu, highs = (w[t] >> 4) & 0x0F0F0F0Fu;
          q[2 * t] = __hsub2(bits_h2(__byte_perm(lows, 0x64646464u, 0x4140)), zp), q[2 * t + 1] = __hsub2(bits_h2(__byte_perm(lows, 0x64646464u, 0x4342)), zp);
          q[8 + 2 * t] = __hsub2(bits_h2(__byte_perm(highs, 0x64646464u, 0x4140)), zp), q[8 + 2 * t + 1] = __hsub2(bits_h2(__byte_perm(highs, 0x64646464u, 0x4342)), zp);
        }
      }
    };
    // [0, 16): hi = f16(d * q), [16, 32): lo = d * q - hi, exact
    auto scale_up = [&](const __half2 (&q)[16], uint32_t scale, uint32_t (&v)[32]) {
      const __half2 dd = __half2half2(half ? __high2half(bits_h2(scale)) : __low2half(bits_h2(scale)));
#pragma unroll
      for (int c = 0; c < 16; c++) {
        const __half2 h = __hmul2(dd, q[c]);
        v[c] = h2_bits(h), v[16 + c] = h2_bits(__hfma2(dd, q[c], __hneg2(h)));
      }
    };
    for (uint32_t item = item_beg; item < n_items && ok; item += item_step) {
      if (!next_item(item, pstart, pcount)) continue;
      for (uint32_t grp = groups + ((groups ^ team) & 1); grp < groups + n_groups && ok; grp += 2) {
        const uint32_t stage = grp % RAW_STAGES;
        if (!ready) ok = mbar_wait(&raw_full[stage], (grp / RAW_STAGES) & 1);
        __syncwarp();
        uint32_t w[RAW_WORDS], w1[RAW_WORDS], scale, scale1, v[32];
        load(tile0 + stage * RAW_BYTES, mine, w, scale);
        load(tile0 + stage * RAW_BYTES, mine + 1, w1, scale1);
        __half2 q0[16], q1[16];
        integers(w, q0);
        scale_up(q0, scale, v);
        if (EARLY) integers(w1, q1);
        // The first block is converted, and the second as far as registers go, ahead of the wait: that is then off the cycle of MMAs -> done -> store
        // -> MMAs.  Q4_0: its integers (its raw words only: 536 us for 528 on 256 tokens and 8 experts of 4096 x 14336).  Q8_0: its raw words (its integers
        // spill 8 bytes: 256 tokens on 128 experts of 2048 x 768 209 us for 205, on 64 of 2048 x 1408 195 for 193).
#pragma unroll
        for (int i = 0; i < 32; i++) asm volatile("" : "+r"(v[i]));
#pragma unroll
        for (int i = 0; i < (EARLY ? 16 : 0); i++) asm volatile("" : "+r"(*reinterpret_cast<uint32_t *>(&q1[i])));
#pragma unroll
        for (int i = 0; i < (EARLY ? 0 : RAW_WORDS); i++) asm volatile("" : "+r"(w1[i]));
        asm volatile("" : "+r"(scale1));
        __syncwarp();
        if (lane == 0) mbar_arrive(&raw_empty[stage]);
        ready = mbar_test(&raw_full[(grp + 2) % RAW_STAGES], ((grp + 2) / RAW_STAGES) & 1);
        if (grp >= A_RING && ok) {
          // the group's A stages were last read by the MMAs of the group A_RING before it
          const uint32_t sp = grp - A_RING;
          ok = mbar_wait_tmem(&done[sp % DONE_RING], (sp / DONE_RING) & 1);
        }
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        const uint32_t a = a_tmem + grp % A_RING * GROUP * A_STAGE_COLS;
        tc_st32(a, v);
        if (!EARLY) integers(w1, q1);
        scale_up(q1, scale1, v);
        tc_st32(a + A_STAGE_COLS, v);
        tc_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_tmem(leader_addr(&a_full[grp % FULL_RING]));
        ready = __all_sync(0xffffffffu, ready);
      }
      groups += n_groups;
    }
    if (!ok && lane == 0) *s_abort = 1, atomicOr(d.status, MER_DEVSTAT_TIMEOUT);
  } else {
    // ---------------------------------------------------------------------------- epilogue
    // Two groups of four warps, one per accumulator buffer: group e drains the items whose running number is e mod 2,
    // so the epilogues of two consecutive items may overlap each other as well as the MMAs that follow.
    const uint32_t q = warp & 3;         // a warp reads the TMEM lanes 32 * (warp % 4) ..
    const uint32_t row = q * 32 + lane;  // row of the item's 128-row tile
    const uint32_t buf = (warp - W_EPI0) >> 2, gw = (warp - W_EPI0) & 3;  // group, warp within the group
    float *s_un = reinterpret_cast<float *>(smem + 1024 + buf * 2048 + 512);
    float **s_row = reinterpret_cast<float **>(smem + 1024 + buf * 2048 + 1024);  // down phase: each token's output row
    uint32_t next_buf = 0, used = 0;  // buffer of the next resident item that takes one; uses of this group's
    // A group whose bounded wait expired goes "dead": it stops touching TMEM and waiting but keeps walking the items, so
    // that the group's named barriers always see all four warps.
    bool dead = false;
    for (uint32_t item = item_beg; item < n_items; item += item_step) {
      const uint32_t mt = (item % m_pairs) * PAIR + rank;
      const bool resident = next_item(item, pstart, pcount, &split) != nullptr;
      // A wide item fills both buffers, and each group drains its own.
      const bool wide = pcount > BUF_TOKENS;
      const uint32_t col0 = wide ? buf * BUF_TOKENS : 0, cols = min(pcount - col0, BUF_TOKENS);  // this group's columns of the pass
      if (resident) {
        const uint32_t which = next_buf;
        next_buf = wide ? 0 : which ^ 1;
        if (!wide && which != buf) continue;  // the other group's item
      } else if (!wide && buf != 0) {
        continue;  // narrow items of missing experts are zero-filled by group 0
      }
      // The pass's pair indices and un-scale factors go to shared memory (one column per thread of the group), fetched
      // before the accumulator is waited for so that their latency hides behind the item's MMAs; the column loop then
      // reads them as broadcasts.
      {
        const uint32_t c = gw * 32 + lane;
        const bool have = c < cols;
        const float un = have ? __ldg(p.unscale + pstart + col0 + c) : 0.0f;
        asm volatile("bar.sync %0, 128;" ::"r"(1 + buf) : "memory");  // the group has finished reading the previous item's tables
        s_un[c] = un;
        if (p.phase == 1) s_row[c] = have ? pair_output_row(d, p.out, __ldg(d.perm + pstart + col0 + c)) : nullptr;
        asm volatile("bar.sync %0, 128;" ::"r"(1 + buf) : "memory");
      }
      if (resident && !dead) {
        ok = mbar_wait_tmem(&acc_full[buf], used & 1);
        used++;
        if (*s_abort) ok = false;
        if (!__all_sync(0xffffffffu, ok)) dead = true;
        tc_fence_after();
      } else if (!resident && warp == W_EPI0 && lane == 0) {
        atomicOr(d.status, MER_DEVSTAT_RESIDENCY_MISS);  // fail closed: zeros below
      }
      const uint32_t acc_addr = tmem_base + ((q * 32u) << 16) + buf * 128;
      const bool is_gate = (lane & 8) == 0;
      const bool clamp = d.swiglu_limit > 0.0f && isfinite(d.swiglu_limit);
      constexpr int EC = 16;  // columns (tokens) at a time
      for (uint32_t cbase = 0; cbase < cols && mt < m_tiles; cbase += EC) {
        float val[EC];
        if (resident && !dead) {
          uint32_t v[EC];
          tc_ld16(acc_addr + cbase, v);
#pragma unroll
          for (int i = 0; i < EC; i++) val[i] = __uint_as_float(v[i]);
          if (split) {
            tc_ld16(acc_addr + SPLIT_TOKENS + cbase, v);
#pragma unroll
            for (int i = 0; i < EC; i++) val[i] += __uint_as_float(v[i]);
          }
        } else {
#pragma unroll
          for (int i = 0; i < EC; i++) val[i] = 0.0f;
        }
        // the steps run column-batched (all multiplies, then all shuffles, ...): warp-synchronous operations are kept in
        // program order, so a column-by-column loop would serialise on the latency of every single one
#pragma unroll
        for (int i = 0; i < EC; i += 4) {
          const float4 un = *reinterpret_cast<const float4 *>(s_un + cbase + i);
          val[i] *= un.x, val[i + 1] *= un.y, val[i + 2] *= un.z, val[i + 3] *= un.w;
        }
        if (p.phase == 0) {
          // rows come in packed tiles of 16: slots 0..7 gate rows, 8..15 the matching up rows.  The two lanes of a
          // gate/up pair exchange halves: the gate lane finishes the first eight columns, the up lane the others.
          float h[EC / 2];
#pragma unroll
          for (int i = 0; i < EC / 2; i++) h[i] = __shfl_xor_sync(0xffffffffu, is_gate ? val[EC / 2 + i] : val[i], 8);
#pragma unroll
          for (int i = 0; i < EC / 2; i++) {
            float gate = is_gate ? val[i] : h[i];
            const float up = is_gate ? h[i] : val[EC / 2 + i];
            if (clamp && gate == gate) gate = fminf(fmaxf(gate, -d.swiglu_limit), d.swiglu_limit);
            h[i] = __fdividef(gate, 1.0f + __expf(-gate)) * up;
          }
          // h in the order of the groups: its rows are then the rows of the down phase's passes
          const uint32_t col = cbase + (is_gate ? 0 : EC / 2);
          float *dst = p.out + (size_t)(pstart + col0 + col) * d.F + (mt * 8 + (row >> 4)) * 8 + (lane & 7);
#pragma unroll
          for (int i = 0; i < EC / 2; i++)
            if (col + i < cols) dst[(size_t)i * d.F] = h[i];
        } else {
          const uint32_t off = mt * 128 + row;
#pragma unroll
          for (int i = 0; i < EC; i++)
            if (cbase + i < cols) s_row[cbase + i][off] = val[i];
        }
      }
      if (resident && !dead) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_tmem(leader_addr(&acc_empty[buf]));
      }
    }
    if (dead && lane == 0) *s_abort = 1, atomicOr(d.status, MER_DEVSTAT_TIMEOUT);
  }

  // neither CTA may leave while the other's MMAs read its memory or its warps signal barriers here
  tc_fence_before();
  cluster_sync();
  if (warp == W_MMA) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

// Four values of a row -> their hi and lo parts.
__device__ __forceinline__ void split_values(float4 v, float sc, uint2 &hi, uint2 &lo) {
  const float a = v.x * sc, b = v.y * sc, c = v.z * sc, e = v.w * sc;
  const __half2 h0 = __floats2half2_rn(a, b), h1 = __floats2half2_rn(c, e);
  const float2 f0 = __half22float2(h0), f1 = __half22float2(h1);
  hi = make_uint2(h2_bits(h0), h2_bits(h1));
  lo = make_uint2(h2_bits(__floats2half2_rn(a - f0.x, b - f0.y)), h2_bits(__floats2half2_rn(c - f1.x, e - f1.y)));
}

// Rows of activations -> their f16 hi parts and lo parts (act_rows.h: `rows` of them), after an exact power-of-two scaling of the
// row, and its inverse.  Row i of the output belongs to the i-th pair in group order, so that a pass is a run of rows and
// one copy fetches a chunk of all of them.  The source is row i of h, the row of pair i's token with `perm`, or with `pos` the tokens' rows: a row is then read and
// converted once and written to the places of all of its `slots` pairs (rows picked by the GEMM's own copies instead, four per gather, took 80 cycles per four
// rows and doubled the GEMM's time).  TPR threads per row.  What bounds it is writing the rows.  With a row of x read and converted by each of
// its pairs: 4096 tokens of 7168 for nine experts each 299 us.  Three blocks an SM: without that bound the places' addresses take 122 registers instead of 54.
template <int TPR, bool TOKENS>
__global__ void __launch_bounds__(256, 3) k_split_rows(const float *__restrict__ act, uint32_t n_rows, uint32_t K, const uint32_t *__restrict__ pos,
                                                    const uint32_t *__restrict__ perm, uint32_t slots, const uint32_t *__restrict__ n_grouped, uint2 *__restrict__ out,
                                                    uint32_t rows, float *__restrict__ unscale) {
  const uint32_t i = blockIdx.x * (256 / TPR) + threadIdx.x / TPR, t = threadIdx.x % TPR;
  const bool have = TOKENS ? i < n_rows : i < *n_grouped;  // fewer than the pairs of the dispatch under expert parallelism
  if (TPR <= 32 && !have) return;
  const float4 *src = reinterpret_cast<const float4 *>(act + (size_t)(!have ? 0 : !TOKENS && perm ? __ldg(perm + i) / slots : i) * K);
  float mx = 0.0f;
  bool nan = false;
  if (have) {
#pragma unroll 4
    for (uint32_t k = t; k < K / 4; k += TPR) {
      const float4 v = __ldg(src + k);
      nan |= (v.x != v.x) | (v.y != v.y) | (v.z != v.z) | (v.w != v.w);
      mx = fmaxf(fmaxf(fmaxf(fmaxf(mx, fabsf(v.x)), fabsf(v.y)), fabsf(v.z)), fabsf(v.w));
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (__any_sync(0xffffffffu, nan)) mx = __uint_as_float(0x7fc00000u);
  if (TPR > 32) {
    __shared__ float s_mx[8];
    if ((threadIdx.x & 31) == 0) s_mx[threadIdx.x >> 5] = mx;
    __syncthreads();
    mx = s_mx[0];
    for (int w = 1; w < 8; w++) mx = s_mx[w] != s_mx[w] || mx != mx ? __uint_as_float(0x7fc00000u) : fmaxf(mx, s_mx[w]);
    if (!have) return;
  }
  float sc = 1.0f;
  if (mx > 0.0f && isfinite(mx)) {
    int e;
    frexpf(mx, &e);
    sc = ldexpf(1.0f, (int)POW2_SCALE_TARGET - e);  // mx * sc in [256, 512)
  } else if (mx != mx || isinf(mx)) {
    sc = mx;  // non-finite activations poison the row, as they would in fp32
  }
  const size_t lo_part = act_rows_lo(rows);
  if (!TOKENS) {
    if (t == 0) unscale[i] = 1.0f / sc;
#pragma unroll 4
    for (uint32_t k = t; k < K / 4; k += TPR) {
      uint2 *dst = out + act_rows_hi(rows, i, k);
      split_values(__ldg(src + k), sc, dst[0], dst[lo_part]);
    }
    return;
  }
  constexpr uint32_t S = 9, U = 4;  // places a pass over the row writes to; steps of it in flight
#pragma unroll 1
  for (uint32_t s0 = 0; s0 < slots; s0 += S) {
    uint32_t at[S];
#pragma unroll
    for (uint32_t j = 0; j < S; j++) {
      at[j] = s0 + j < slots ? __ldg(pos + (size_t)i * slots + s0 + j) : MER_NONE;
      if (t == 0 && at[j] != MER_NONE) unscale[at[j]] = 1.0f / sc;
    }
#pragma unroll 1
    for (uint32_t k0 = t; k0 < K / 4; k0 += U * TPR) {
      float4 v[U];
#pragma unroll
      for (uint32_t u = 0; u < U; u++) v[u] = k0 + u * TPR < K / 4 ? __ldg(src + k0 + u * TPR) : make_float4(0, 0, 0, 0);
#pragma unroll
      for (uint32_t u = 0; u < U; u++) {
        const uint32_t k = k0 + u * TPR;
        if (k >= K / 4) break;
        uint2 hi, lo;
        split_values(v[u], sc, hi, lo);
        uint2 *first = out + act_rows_hi(rows, 0, k), *first_lo = first + lo_part;
#pragma unroll
        for (uint32_t j = 0; j < S; j++)
          if (at[j] != MER_NONE) first[at[j] * ACT_ROW] = hi, first_lo[at[j] * ACT_ROW] = lo;
      }
    }
  }
}

void launch_split_rows(const float *act, uint32_t n_rows, uint32_t K, const uint32_t *pos, const uint32_t *perm, uint32_t slots, const uint32_t *n_grouped,
                       uint2 *out, uint32_t rows, float *unscale, cudaStream_t s) {
  // a warp per row keeps short rows of large batches cheap; long rows, and few of them, want more loads in flight
  const bool warps = K <= 2048 && n_rows >= 2048;
  auto kern = pos ? (warps ? k_split_rows<32, true> : k_split_rows<256, true>) : (warps ? k_split_rows<32, false> : k_split_rows<256, false>);
  kern<<<warps ? (n_rows + 7) / 8 : n_rows, 256, 0, s>>>(act, n_rows, K, pos, perm, slots, n_grouped, out, rows, unscale);
}

using EncodeTiled = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                 const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
// The driver's encoder, looked up once; null when the driver has none.
EncodeTiled encode_tiled() {
  static const EncodeTiled fn = [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    const cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q);
    return e == cudaSuccess && q == cudaDriverEntryPointSuccess ? reinterpret_cast<EncodeTiled>(p) : nullptr;
  }();
  return fn;
}
// Rows past the end read as zeros.
bool activation_maps(ActMaps *maps, void *base, uint32_t rows, uint32_t K) {
  const EncodeTiled fn = encode_tiled();
  bool ok = fn != nullptr;
  for (uint32_t i = 0; i < PASS_TOKENS / 16 && ok; i++) {
    const ActMapShape a(rows, K, 8 * (i + 1), CHUNKS);
    const cuuint32_t step[4] = {1, 1, 1, 1};
    ok = fn(&maps->m[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, base, a.dims, a.strides, a.box, step, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  }
  return ok;
}

struct GemmPlan {
  uint32_t n_b;
  size_t smem;
};

GemmPlan gemm_plan(int dtype) {
  const uint32_t tile_raw = RAW_BLOCKS * 16 * (dtype == MER_DTYPE_Q4_0 ? MER_Q4_BLOCK_BYTES : MER_Q8_BLOCK_BYTES);
  GemmPlan pl{};
  pl.n_b = 4;  // activation stages of one group
  pl.smem = G_HEADER + (size_t)RAW_STAGES * 8 * tile_raw + (size_t)pl.n_b * B_STAGE;
  return pl;
}

size_t unscale_bytes(uint32_t max_pairs) { return ((size_t)max_pairs * 4 + 255) & ~(size_t)255; }

}  // namespace

bool gemm_ffn_supported(int dtype, uint32_t D, uint32_t F) {
  return (dtype == MER_DTYPE_Q4_0 || dtype == MER_DTYPE_Q8_0) && D % 128 == 0 && F % 128 == 0;  // whole 128-row tiles, whole weight stages
}

// Scales and split rows of the pairs, for gate/up and then for down.
size_t gemm_ffn_scratch_bytes(uint32_t max_pairs, uint32_t D, uint32_t F) {
  return unscale_bytes(max_pairs) + (size_t)max_pairs * (D > F ? D : F) * 4;
}

// Tokens per pass at most, or 0 when the dispatch is better served by the streaming kernels.
uint32_t gemm_pick_bn(const MoeDispatch &d, uint32_t min_mean_tokens, int sm_count) {
  const uint64_t P = (uint64_t)d.n_tokens * d.slots;
  const uint32_t groups = d.active_groups_hint ? d.active_groups_hint : 1;
  const uint64_t mean = (d.expected_pairs ? d.expected_pairs : P) / groups;
  if (mean < min_mean_tokens || P > d.scratch_pairs) return 0;
  // Passes of up to 256 tokens instead of 128 save conversions of the weights (129 to 256 tokens of an expert: half of them) and leave the MMAs idle while
  // an item's epilogue drains both buffers, some 5000 cycles.  That pays where an item's K is long and where there are enough items to
  // share out evenly.  Us a pass, 128 / 256: 4096 tokens on 256 experts of 7168 x 2048 8490 / 8340; 2 layers of 2048 on 128 of 2048 x 768 (24 blocks of K
  // in the down phase) 1053 / 1226; 256 on 8 of 4096 x 14336 (two items a pair of CTAs in the down phase) 528 / 582.  Beside the line of K, 200 tokens each: 64 experts
  // of 2048 x 1536 624 / 786, of 4096 x 1536 with Zipf routing 1224 / 1300.  Below the line of items (five to seven a pair) it depends on how
  // the experts' tokens fill passes: 2 layers of 32 of 4096 x 2048, 200 each, 1540 / 1500; 32 of 4096 x 8192, 162 each, 2590 / 2520.
  const bool long_k = d.D / 32 >= 128 && d.F / 32 >= 64, many = (uint64_t)groups * (std::min(2 * d.F, d.D) / 256) >= 8 * (uint64_t)(sm_count / PAIR);
  return long_k && many ? PASS_TOKENS : BUF_TOKENS;
}

void gemm_bind(MoeDispatch &d, void *stream_scratch, int sm_count, uint32_t bn) {
  stream_bind(d, stream_scratch, sm_count, true);  // pass tables live in the streaming scratch
  d.tokens_per_pass = bn;
  d.item_bounds = nullptr;  // items are dealt round-robin
  d.pass_desc = nullptr, d.x_rows = nullptr, d.taken = nullptr;
}

cudaError_t launch_ffn_gemm(MoeDispatch &d, void *scratch, size_t scratch_bytes, int sm_count, cudaStream_t s, int *launches, cudaEvent_t ev_mid) {
  const GemmPlan pl = gemm_plan(d.dtype);
  const uint32_t P = d.n_tokens * d.slots;
  float *unscale = reinterpret_cast<float *>(scratch);
  const size_t off = unscale_bytes(d.scratch_pairs);
  uint2 *rows = reinterpret_cast<uint2 *>(static_cast<uint8_t *>(scratch) + off);
  if (P > d.scratch_pairs || off + (size_t)P * (d.D > d.F ? d.D : d.F) * 4 > scratch_bytes) return cudaErrorInvalidConfiguration;
  auto kern = d.dtype == MER_DTYPE_Q4_0 ? k_ffn_gemm<MER_DTYPE_Q4_0> : k_ffn_gemm<MER_DTYPE_Q8_0>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pl.smem);
  if (e != cudaSuccess) return e;

  for (int phase = 0; phase < 2; phase++) {
    const uint32_t K = phase == 0 ? d.D : d.F;
    // Under expert parallelism few of a token's pairs are here, of many tokens none: each pair's row by itself (512 tokens from each of 16 ranks, 16 of 256 experts of
    // 4096 x 1536 here: 274 us a layer by token).
    const bool by_token = phase == 0 && d.expected_pairs == 0;
    launch_split_rows(phase == 0 ? d.x : d.h, by_token ? d.n_tokens : P, K, by_token ? d.pos : nullptr, phase == 0 ? d.perm : nullptr, d.slots, d.offsets + d.n_groups, rows,
                      P, unscale, s);
    ActMaps maps;
    if (!activation_maps(&maps, rows, P, K)) return cudaErrorNotSupported;
    GemmParams p{};
    p.d = d, p.phase = phase, p.unscale = unscale;
    p.rows = phase == 0 ? d.F : d.D;
    p.kb_total = K / 32;
    p.n_b = pl.n_b;
    p.out = phase == 0 ? d.h : d.y;
    kern<<<sm_count / PAIR * PAIR, G_THREADS, pl.smem, s>>>(p, maps);
    if (phase == 0 && ev_mid) cudaEventRecord(ev_mid, s);
  }
  d.y_parts = nullptr, d.y_nparts = 1;
  if (launches) (*launches) += 4;
  return cudaGetLastError();
}
