// Attention of prompts on the 5th-generation tensor cores, two query tiles per CTA:
//   * staircase attention over packed sequences (a query row sees the keys up to the right edge of its right-aligned block;
//     nanovllm/kernels/triton/attention/block_prefill_attention_v2.py:17-166);
//   * window attention of prompt portions over the paged KV cache (WIN, stairs of one token: a query row sees the last
//     `window` keys up to its own), with an optional sink in the softmax's denominator, one output gate per head, and heads of
//     64 or 128 stored channels.
//
// A tile is 128 query rows, `tokens x group` of one sequence and KV head (row = token * group + head in group); a unit is two
// neighbouring tiles A and B of one sequence, which walk the same key tiles of 128 keys.  Roles: a TMA warp (both Q tiles, K and
// V rings), an MMA warp, and four softmax warps per tile, one query row per thread.
//
// What bounds it: the chain of a tile (S ready, scores to registers, maximum, exponentials, P back, P V) took 1.7 us for
// 128 keys and 0.27 us of products while one tile had the SM to itself.  Here one tile's softmax runs under the other's products,
// and P goes back into the tensor memory of the scores it came from (bf16 pairs, the left operand of P V): no shared memory for P
// and no proxy fence.  The products of one thread run in the order of issue, so new scores may follow P V into the same columns
// without a wait.  A unit of one tile (see the launch) takes both score buffers in turn, the next scores ahead of P V.
// 4 x 4096 tokens, 16 query and 8 KV heads: 400 -> 289 us alone, 417 -> 333 - 337 in a loop at the power limit, the same bits.  (Steps of
// 64 keys with two score buffers per tile and an issuing warp per tile: 299 us alone, 329 in a loop, other roundings; an issuing
// warp per tile with these steps: 351.)
//
// Tensor memory: S_A (P_A) | S_B (P_B) | O_A | O_B, 128 columns each; with one tile S of even key tiles | - | O | S of odd ones.
#include "mdb_common.cuh"

namespace mdb {

// Times of a unit, in sixteenths of a key tile of one query tile: a key tile, and the start and end of a unit.  Fitted to both forms'
// times of 100 calls (one to 64 prompts of 64 to 4096 tokens, alike and not); the worst choice left is 11 % off the better.
constexpr int kApTileStep = 16, kApTileUnit = 32, kApPairStep = 23, kApPairUnit = 32;

struct ApPlan {
  static constexpr int kKStages = 3, kVStages = 2;
  static constexpr int kQBytes = 2 * 128 * 128;             // a tile: two channel halves of [128 rows][128 B]
  static constexpr int kThreads = 384;                      // three warpgroups; two warps idle
  // registers: 384 threads x 168 at launch = 256 x 216 (softmax) + 128 x 72, no spills (208 / 88: 291 against 289 us)
  static constexpr int kSoftmaxRegs = 216, kOtherRegs = 72;
  static_assert(256 * kSoftmaxRegs + 128 * kOtherRegs <= kThreads * 168, "registers after the split");
  static constexpr int kOffK = 2 * kQBytes;
  static constexpr int kOffV = kOffK + kKStages * kAtTileBytes;
  static constexpr int kOffBars = kOffV + kVStages * kAtTileBytes;
  static constexpr int kOffList = kOffBars + 256;            // the sorted list of items
  static constexpr int kMaxItems = 256, kMaxSeqs = 1024;
  static constexpr int kSmemBytes = 1024 + kOffList + kMaxItems * 4;
};
static_assert(ApPlan::kSmemBytes <= 227 * 1024, "shared memory of the prompt attention");

// The softmax warps, four for every tile there may be, then the other roles.
template <bool DEAL>
struct ApRoles {
  static constexpr int kProducer = DEAL ? 8 : 4, kMma = DEAL ? 9 : 5, kThreads = DEAL ? ApPlan::kThreads : 192;
};

// barrier slots; those of a tile (A, B) come in pairs, those of a score buffer in threes
enum {
  kApBarQFull = 0, kApBarQEmpty = 1, kApBarQReady = 2, kApBarKFull = 4, kApBarKEmpty = 7, kApBarVFull = 10, kApBarVEmpty = 12,
  kApBarSFull = 14, kApBarPFull = 17, kApBarPDone = 20, kApBarOFull = 22, kApBarOEmpty = 24, kApBarCount = 26
};
// Score buffers: of tile A, of tile B, and the second one of a unit without tile B, in B's output columns
constexpr int kApAlone = 2;
__device__ __forceinline__ uint32_t ap_score_col(int buf) { return buf == kApAlone ? 384u : 128u * buf; }

// Four products in a row with one elected lane: left operand steps of `a_step`, right operand steps of `b_step` (descriptor
// units of 16 bytes).
__device__ __forceinline__ void umma_bf16_x4_w(uint32_t d_tmem, uint64_t a_desc, uint64_t a_step, uint64_t b_desc, uint64_t b_step, uint32_t idesc,
                                               uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, t, q;\n\t.reg .b64 a1, a2, a3, b1, b2, b3;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "setp.ne.b32 p, %4, 0;\n\tsetp.eq.b32 t, 0, 0;\n\t"
      "add.u64 a1, %1, %5;\n\tadd.u64 a2, a1, %5;\n\tadd.u64 a3, a2, %5;\n\t"
      "add.u64 b1, %2, %6;\n\tadd.u64 b2, b1, %6;\n\tadd.u64 b3, b2, %6;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a1, b1, %3, t;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a2, b2, %3, t;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a3, b3, %3, t;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "l"(a_step), "l"(b_step)
      : "memory");
}
// ... with the left operand in tensor memory: bf16 pairs, one row per lane, eight columns per step
__device__ __forceinline__ void umma_bf16_ts_x4_w(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint64_t b_step, uint32_t idesc,
                                                  uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, t, q;\n\t.reg .b64 b1, b2, b3;\n\t.reg .b32 a1, a2, a3;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "setp.ne.b32 p, %4, 0;\n\tsetp.eq.b32 t, 0, 0;\n\t"
      "add.u32 a1, %1, 8;\n\tadd.u32 a2, %1, 16;\n\tadd.u32 a3, %1, 24;\n\t"
      "add.u64 b1, %2, %5;\n\tadd.u64 b2, b1, %5;\n\tadd.u64 b3, b2, %5;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a1], b1, %3, t;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a2], b2, %3, t;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a3], b3, %3, t;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate), "l"(b_step)
      : "memory");
}
struct ApTile {
  bool valid;
  int m0;             // first query
  int end;            // keys in front of it are seen by a row of the tile
  int first, last;    // key tiles [first, last) of the unit
};
struct ApUnit {
  int seq, kvh, q_start, Tq, q_off, T, seq_start;
  int kbeg, ntiles;      // ntiles 0: nothing to do
  int cut;               // window form: key tile inside which tile A's keys end and B's go on (-1: none)
  ApTile t[2];
};

// Where a sequence's queries and keys lie.
struct ApSeq {
  int q_start, Tq, q_off, T, seq_start;
};
template <bool WIN>
__device__ __forceinline__ ApSeq ap_seq(const AtArgs& a, int seq) {
  ApSeq w = {};
  const int32_t* cu_q = a.cu_seqlens_q != nullptr ? a.cu_seqlens_q : a.cu_seqlens;
  w.q_start = cu_q[seq];
  w.Tq = cu_q[seq + 1] - w.q_start;
  if (WIN) {
    w.q_off = a.start[seq];
    w.T = w.q_off + w.Tq;
  } else {
    w.seq_start = a.cu_seqlens[seq];
    w.T = a.cu_seqlens[seq + 1] - w.seq_start;
    w.q_off = w.T - w.Tq;
  }
  return w;
}
// Keys [x, y) that the rows of the query tile from query m0 on see.
template <bool WIN>
__host__ __device__ __forceinline__ int2 ap_keys(const AtArgs& a, const ApSeq& w, int m0) {
  const int S = 1 << a.log2_stairs;
  const int pad = ((w.T + S - 1) >> a.log2_stairs << a.log2_stairs) - w.T;
  const int last = w.q_off + min(m0 + a.tokens_per_unit, w.Tq) - 1;
  return make_int2(WIN && a.window > 0 ? max(0, w.q_off + m0 - a.window + 1) : 0,
                   min(w.T, ((((last + pad) >> a.log2_stairs) + 1) << a.log2_stairs) - pad));
}

// How the units of a launch are dealt out: `tiles` query tiles each; either the sorted list of `items` (sequence, tile or pair) for
// every KV head, or (items 0) all that the longest sequence allows for, the late ones first.
struct ApDeal {
  int tiles, items, units;
};
// Time of a unit of the query tiles from tile `first` on.
template <bool WIN>
__host__ __device__ __forceinline__ int ap_cost(const AtArgs& a, const ApSeq& w, int first, bool pair) {
  const int m0 = first * a.tokens_per_unit, m1 = m0 + a.tokens_per_unit;
  pair = pair && m1 < w.Tq;
  const int2 k0 = ap_keys<WIN>(a, w, m0);
  const int end = pair ? ap_keys<WIN>(a, w, m1).y : k0.y, steps = (end + kAtKeys - 1) / kAtKeys - k0.x / kAtKeys;
  return pair ? kApPairStep * steps + kApPairUnit : kApTileStep * steps + kApTileUnit;
}

// Where the sequences differ, by all threads: picks tiles alone or pairs and sorts the units by their time, so that dealing them in
// alternating direction gives every CTA about the same.  Sequences of few queries and many keys beside prompts, and batches
// in which one sequence is the longest by far, would leave the list of all that is possible nearly empty and its order the wrong
// one (8 sequences, a prompt of 512 tokens and 7 rows behind 4000 keys: 103 us unsorted in pairs, 59 us; [1000] and 40 times 60
// tokens 57 -> 36 us).  It takes 1.2 us.  `answer`: two words of shared memory; `scratch`: memory of the operand tiles, not in use yet.
template <bool WIN>
__device__ __forceinline__ ApDeal ap_deal(const AtArgs& a, int* answer, uint32_t* scratch, uint32_t* list) {
  const int tid = threadIdx.x, lane = tid & 31, G = static_cast<int>(gridDim.x);
  int* const first_item = reinterpret_cast<int*>(scratch); // [nseq]
  uint32_t* const keys = scratch + ApPlan::kMaxSeqs;
  auto tiles_of = [&](const ApSeq& w) { return min(a.max_qtiles, (max(w.Tq, 0) + a.tokens_per_unit - 1) / a.tokens_per_unit); };
  const int per_rank = a.nseq * a.hkv;
  if (a.tiles_per_unit > 0) return {a.tiles_per_unit, 0, (a.max_qtiles + a.tiles_per_unit - 1) / a.tiles_per_unit * per_rank};
  if (tid < 32) {
    // tiles of the sequences, their time in all, its extremes; the same in pairs
    int v[8] = {0, 0, 0, 0x7fffffff, 0, 0, 0, 0x7fffffff};
    for (int s = lane; s < a.nseq; s += 32) {
      const ApSeq w = ap_seq<WIN>(a, s);
      const int nt = tiles_of(w), np = (nt + 1) / 2;
      if (s < ApPlan::kMaxSeqs) first_item[s] = nt;
      if (nt > 0) {
        const int t0 = ap_cost<WIN>(a, w, 0, false), t1 = ap_cost<WIN>(a, w, nt - 1, false);
        const int p0 = ap_cost<WIN>(a, w, 0, true), p1 = ap_cost<WIN>(a, w, 2 * np - 2, true);
        v[0] += nt; v[1] += nt * ((t0 + t1) / 2); v[2] = max(v[2], max(t0, t1)); v[3] = min(v[3], min(t0, t1));
        v[4] += np; v[5] += np * ((p0 + p1) / 2); v[6] = max(v[6], max(p0, p1)); v[7] = min(v[7], min(p0, p1));
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
      v[i] = (i & 3) < 2 ? __reduce_add_sync(0xffffffffu, v[i]) : (i & 3) == 2 ? __reduce_max_sync(0xffffffffu, v[i]) : __reduce_min_sync(0xffffffffu, v[i]);
    // units of equal times take whole rounds; the more they differ, the better the rounds even out
    auto time = [&](int n, int all, int most, int least) {
      const float rounds = fmaxf(n, 1) * a.hkv / G, alike = most > 0 ? static_cast<float>(least) / most : 1.f;
      return fmaxf(most, all / fmaxf(n, 1) * (rounds + alike * (ceilf(rounds) - rounds)));
    };
    const int per = time(v[0], v[1], v[2], v[3]) <= time(v[4], v[5], v[6], v[7]) ? 1 : 2;
    const int items = per == 1 ? v[0] : v[4];
    const bool sorted = a.nseq <= ApPlan::kMaxSeqs && items <= ApPlan::kMaxItems;
    if (lane == 0) { answer[0] = per; answer[1] = sorted ? items : 0; }
    int before = 0;
    for (int s0 = 0; sorted && s0 < a.nseq; s0 += 32) {
      const int s = s0 + lane, mine = s < a.nseq ? (first_item[s] + per - 1) / per : 0;
      int upto = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += up;
      }
      if (s < a.nseq) first_item[s] = before + upto - mine;
      before += __shfl_sync(0xffffffffu, upto, 31);
    }
  }
  __syncthreads();
  const int per = answer[0], items = answer[1];
  uint32_t item = 0, key = 0;
  if (tid < items) {
    int lo = 0, hi = a.nseq;                               // the last sequence whose first item is not behind this one
    while (hi - lo > 1) {
      const int mid = (lo + hi) / 2;
      if (first_item[mid] <= tid) lo = mid;
      else hi = mid;
    }
    // (of sequences without items the one behind them has the same first item, and is the later one)
    const int at = tid - first_item[lo];
    item = static_cast<uint32_t>(lo) << 16 | static_cast<uint32_t>(at);
    key = static_cast<uint32_t>(min(ap_cost<WIN>(a, ap_seq<WIN>(a, lo), at * per, per == 2), 0xffffff)) << 8 | static_cast<uint32_t>(255 - tid);
  }
  if (tid < ApPlan::kMaxItems) keys[tid] = key;            // (0: behind all items)
  __syncthreads();
  if (tid < items) {
    int rank = 0;
#pragma unroll 4
    for (int i = 0; i < items; i += 4) {
      const uint4 k = *reinterpret_cast<const uint4*>(keys + i);
      rank += (k.x > key) + (k.y > key) + (k.z > key) + (k.w > key);
    }
    list[rank] = item;
  }
  fence_async_smem();
  __syncthreads();
  return {per, items, items > 0 ? items * a.hkv : (a.max_qtiles + per - 1) / per * per_rank};
}

// Unit of this CTA in a wave.
template <bool WIN, bool DEAL>
__device__ __forceinline__ ApUnit ap_unit(const AtArgs& a, const ApDeal& deal, const uint32_t* list, int wave) {
  ApUnit w = {};
  w.cut = -1;
  const int G = static_cast<int>(gridDim.x), c = static_cast<int>(blockIdx.x);
  const int p = wave * G + ((wave & 1) ? G - 1 - c : c);
  if (p >= deal.units) return w;
  int at;                                                  // first tile / tiles of a unit
  if (DEAL && deal.items > 0) {
    const uint32_t item = list[p / a.hkv];
    w.seq = static_cast<int>(item >> 16);
    at = static_cast<int>(item & 0xffffu);
    w.kvh = p % a.hkv;
  } else {
    const int per_rank = a.nseq * a.hkv, rest = p % per_rank;
    at = (a.max_qtiles + deal.tiles - 1) / deal.tiles - 1 - p / per_rank;
    w.seq = rest / a.hkv;
    w.kvh = rest % a.hkv;
  }
  const ApSeq q = ap_seq<WIN>(a, w.seq);
  w.q_start = q.q_start; w.Tq = q.Tq; w.q_off = q.q_off; w.T = q.T; w.seq_start = q.seq_start;
#pragma unroll
  for (int x = 0; x < 2; ++x) {
    ApTile& t = w.t[x];
    t.m0 = (deal.tiles * at + x) * a.tokens_per_unit;
    t.valid = x < (DEAL ? deal.tiles : 1) && t.m0 < w.Tq;
    if (!t.valid) continue;
    const int2 keys = ap_keys<WIN>(a, q, t.m0);
    // window form: from the tile of keys that holds the first query's first key
    if (x == 0) w.kbeg = keys.x / kAtKeys * kAtKeys;
    t.end = keys.y;
    t.first = (keys.x - w.kbeg) / kAtKeys;
    t.last = (keys.y - w.kbeg + kAtKeys - 1) / kAtKeys;
    w.ntiles = t.last;
  }
  if (WIN && w.t[1].valid && w.t[0].end < w.kbeg + w.t[0].last * kAtKeys) w.cut = w.t[0].last - 1;
  return w;
}

// DEAL: more tiles than SMs, in sequences of more than one
template <bool WIN, bool DEAL>
__global__ void __launch_bounds__(ApRoles<DEAL>::kThreads, 1)
attn_prompt_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                   const __grid_constant__ CUtensorMap map_v, const AtArgs a, const int units) {
  using P = ApPlan;
  constexpr int kProducerWarp = ApRoles<DEAL>::kProducer, kMmaWarp = ApRoles<DEAL>::kMma;
  const int halves = WIN ? a.halves : 2;      // 64-channel halves of a stored head
  extern __shared__ __align__(1024) unsigned char ap_smem_raw[];
  const uint32_t raw = smem_u32(ap_smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  unsigned char* gen_base = ap_smem_raw + (base - raw);
  const uint32_t bars = base + P::kOffBars;
  auto bar = [&](int slot) { return bars + 8u * static_cast<uint32_t>(slot); };
  volatile uint32_t* misc = reinterpret_cast<volatile uint32_t*>(gen_base + P::kOffBars + 8 * kApBarCount);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int group = a.group;
  const int rows_used = group * a.tokens_per_unit;      // <= 128

  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    for (int s = 0; s < kApBarCount; ++s) {
      const bool by_softmax = s == kApBarQReady || s == kApBarQReady + 1 || (s >= kApBarPFull && s < kApBarPFull + 3) || s >= kApBarOEmpty;
      mbar_init(bar(s), by_softmax ? 4 : 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kMmaWarp) {
    const uint32_t slot = smem_u32(const_cast<uint32_t*>(&misc[0]));
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = misc[0];
  pdl_wait();   // q and the K/V rows of this step come from the preceding kernels
  const uint32_t* const list = reinterpret_cast<const uint32_t*>(gen_base + P::kOffList);
  ApDeal deal = {1, 0, units};
  if (DEAL)
    deal = ap_deal<WIN>(a, reinterpret_cast<int*>(gen_base + P::kOffBars + 8 * kApBarCount + 8), reinterpret_cast<uint32_t*>(gen_base + P::kOffK),
                        reinterpret_cast<uint32_t*>(gen_base + P::kOffList));
  const int waves = (deal.units + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x);

  if (warp >= kProducerWarp) {
    if (DEAL) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(P::kOtherRegs));
    if (warp == kProducerWarp) {
      // ------------------------------------------------------------------ producer
      if (lane == 0) {
        AtRing kr, vr;
        uint32_t q_phase = 0;
        uint32_t pend_k = 0, pend_v = 0, pend_q = 0;          // stages with a copy in flight, and the parity it completes
        uint32_t par_k = 0, par_v = 0, par_q = 0;
        bool ok = true;
        auto load_tile = [&](const CUtensorMap* map, uint32_t tiles0, int full0, int empty0, int stages, AtRing& r,
                             uint32_t& pend, uint32_t& par, int kvh, int token_row) {
          if (!mbar_wait(bar(empty0 + r.stage), r.phase ^ 1)) return false;
          const uint32_t full = bar(full0 + r.stage);
          const uint32_t dst = tiles0 + r.stage * kAtTileBytes;
          mbar_arrive_expect_tx(full, halves * kAtHalfBytes);
          tma_load_2d(dst, map, kvh * 64 * halves, token_row, full);
          if (halves > 1) tma_load_2d(dst + kAtHalfBytes, map, kvh * kHeadDim + 64, token_row, full);
          pend |= 1u << r.stage;
          par = (par & ~(1u << r.stage)) | (r.phase << r.stage);
          r.advance(stages);
          return true;
        };
        for (int wave = 0; wave < waves && ok; ++wave) {
          const ApUnit w = ap_unit<WIN, DEAL>(a, deal, list, wave);
          if (w.ntiles == 0) continue;
          if (!mbar_wait(bar(kApBarQEmpty), q_phase ^ 1)) { ok = false; break; }
          {
            const uint32_t full = bar(kApBarQFull);
            mbar_arrive_expect_tx(full, static_cast<uint32_t>(rows_used) * 128u * halves * (w.t[1].valid ? 2u : 1u));
#pragma unroll
            for (int x = 0; x < 2; ++x) {
              if (!w.t[x].valid) continue;
              const uint32_t dst = base + x * P::kQBytes;
              tma_load_3d(dst, &map_q, 0, w.kvh * group, w.q_start + w.t[x].m0, full);
              if (halves > 1) tma_load_3d(dst + 128 * 128, &map_q, 64, w.kvh * group, w.q_start + w.t[x].m0, full);
            }
            pend_q = 1u;
            par_q = q_phase;
            q_phase ^= 1;
          }
          auto token_row = [&](int tile) {
            const int key0 = w.kbeg + tile * kAtKeys;
            if (!WIN) return w.seq_start + key0;
            int page = key0 / kPage < a.table_stride ? a.block_table[static_cast<int64_t>(w.seq) * a.table_stride + key0 / kPage] : -1;
            if (page < 0 || page >= a.num_pages) {
              report_status(MDB_STATUS_BAD_PAGE);
              page = 0;
            }
            return page * kPage + key0 % kPage;
          };
          for (int j = 0; j < w.ntiles && ok; ++j) {
            ok = load_tile(&map_k, base + P::kOffK, kApBarKFull, kApBarKEmpty, P::kKStages, kr, pend_k, par_k, w.kvh, token_row(j));
            for (int copy = 0; copy < (WIN && j == w.cut ? 2 : 1) && ok; ++copy)
              ok = load_tile(&map_v, base + P::kOffV, kApBarVFull, kApBarVEmpty, P::kVStages, vr, pend_v, par_v, w.kvh, token_row(j));
          }
        }
        if (!ok) {
          report_status(MDB_STATUS_WAIT_TIMEOUT);
          // let the copies already issued land before the CTA gives its shared memory back
          for (int s = 0; s < P::kKStages; ++s) if (pend_k >> s & 1) mbar_wait(bar(kApBarKFull + s), par_k >> s & 1);
          for (int s = 0; s < P::kVStages; ++s) if (pend_v >> s & 1) mbar_wait(bar(kApBarVFull + s), par_v >> s & 1);
          if (pend_q) mbar_wait(bar(kApBarQFull), par_q);
        }
      }
    } else if (warp == kMmaWarp) {
      // ----------------------------------------------------------------- MMA issue (all lanes, one elected)
      // bf16 x bf16 -> fp32, M = 128, N = 128 (or 64 channels); bit 16 set: B operand MN-major
      const uint32_t idesc_s = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(kAtKeys >> 3) << 17) |
                               (static_cast<uint32_t>(128 >> 4) << 24);
      const uint32_t idesc_o = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) |
                               (static_cast<uint32_t>(halves * 8) << 17) | (static_cast<uint32_t>(128 >> 4) << 24);
      AtRing kr, vr;
      uint32_t p_phase = 0 /* bit per score buffer */, o_phase[2] = {0, 0};
      uint32_t qfull_phase = 0;
      bool ok = true;
      for (int wave = 0; wave < waves && ok; ++wave) {
        const ApUnit w = ap_unit<WIN, DEAL>(a, deal, list, wave);
        if (w.ntiles == 0) continue;
        const bool alone = !w.t[1].valid;
        if (WIN) {
          if (!mbar_wait_w(bar(kApBarQFull), qfull_phase)) { ok = false; break; }
          qfull_phase ^= 1;
        } else {
          // staircase form: the softmax warps scale q in place first.  Those of a tile that is not there have only seen it: the
          // next unit's q may not arrive before all have, or they would miss a phase and wait for a later one.
          if (!mbar_wait_w(bar(kApBarQReady), qfull_phase) || (DEAL && !mbar_wait_w(bar(kApBarQReady + 1), qfull_phase))) { ok = false; break; }
          qfull_phase ^= 1;
        }
        auto issue_s = [&](int x, int buf) {           // scores of tile x with the K tile at the ring's position
          const uint32_t q_tile = base + x * P::kQBytes, k_tile = base + P::kOffK + kr.stage * kAtTileBytes;
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            if (WIN && c >= halves) break;
            umma_bf16_x4_w(tmem_base + ap_score_col(buf), umma_desc_sw128(q_tile + c * (128 * 128)), 2, umma_desc_sw128(k_tile + c * kAtHalfBytes), 2,
                           idesc_s, c);
          }
          umma_commit_w(bar(kApBarSFull + buf));
        };
        auto release_k = [&](int j) {
          umma_commit_w(bar(kApBarKEmpty + kr.stage));
          kr.advance(P::kKStages);
          if (j == w.ntiles - 1) umma_commit_w(bar(kApBarQEmpty));
        };
        if (!mbar_wait_w(bar(kApBarKFull + kr.stage), kr.phase)) { ok = false; break; }
        tc_fence_after();
#pragma unroll
        for (int x = 0; x < 2; ++x)
          if (w.t[x].valid && w.t[x].first == 0) issue_s(x, x);
        release_k(0);
        for (int j = 0; j < w.ntiles && ok; ++j) {
          const bool more = j + 1 < w.ntiles;
          bool k_there = false;
          if (alone && more) {
            // the other buffer held the last key tile, whose P V has been issued; or an output of tile B that must have been read out
            if (j == 0 && !mbar_wait_w(bar(kApBarOEmpty + 1), o_phase[1] ^ 1)) { ok = false; break; }
            if (!mbar_wait_w(bar(kApBarKFull + kr.stage), kr.phase)) { ok = false; break; }
            tc_fence_after();
            issue_s(0, j & 1 ? 0 : kApAlone);
            release_k(j + 1);
          }
          if (!mbar_wait_w(bar(kApBarVFull + vr.stage), vr.phase)) { ok = false; break; }
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            if (!w.t[x].valid) continue;
            if (WIN && x == 1 && j == w.cut) {      // B's copy of the values
              umma_commit_w(bar(kApBarVEmpty + vr.stage));
              vr.advance(P::kVStages);
              if (!mbar_wait_w(bar(kApBarVFull + vr.stage), vr.phase)) { ok = false; break; }
            }
            if (j >= w.t[x].first && j < w.t[x].last) {
              const int buf = alone && (j & 1) ? kApAlone : x;
              if (j == w.t[x].first) {
                // the previous unit's accumulator must have been read out
                if (!mbar_wait_w(bar(kApBarOEmpty + x), o_phase[x] ^ 1)) { ok = false; break; }
                o_phase[x] ^= 1;
              }
              if (!mbar_wait_w(bar(kApBarPFull + buf), p_phase >> buf & 1)) { ok = false; break; }
              p_phase ^= 1u << buf;
              tc_fence_after();
              const uint32_t v_tile = base + P::kOffV + vr.stage * kAtTileBytes, p = tmem_base + ap_score_col(buf), o = tmem_base + 256 + x * 128;
              umma_bf16_ts_x4_w(o, p, umma_desc_sw128_mn(v_tile), 128, idesc_o, j > w.t[x].first ? 1u : 0u);
              umma_bf16_ts_x4_w(o, p + 32, umma_desc_sw128_mn(v_tile + 4 * 2048), 128, idesc_o, 1u);
              umma_commit_w(bar(kApBarPDone + x));
              if (j == w.t[x].last - 1) umma_commit_w(bar(kApBarOFull + x));
            }
            if (!alone && more && j + 1 >= w.t[x].first && j + 1 < w.t[x].last) {
              if (!k_there && !mbar_wait_w(bar(kApBarKFull + kr.stage), kr.phase)) { ok = false; break; }
              k_there = true;
              tc_fence_after();
              issue_s(x, x);
            }
          }
          if (!ok) break;
          umma_commit_w(bar(kApBarVEmpty + vr.stage));
          vr.advance(P::kVStages);
          if (!alone && more) release_k(j + 1);      // (the key tiles of A and B overlap or touch: every one is used by a tile)
        }
      }
      if (!ok && lane == 0) report_status(MDB_STATUS_WAIT_TIMEOUT);
    }
  } else {
    // ------------------------------------------------------------------- softmax
    if (DEAL) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(P::kSoftmaxRegs));
    const int x = warp >> 2;                               // tile A or B
    const int row = threadIdx.x & 127;                     // query row of the tile, and its tensor-memory lane
    const int tok_local = row / group, head_in_group = row % group;
    const uint32_t lane_field = static_cast<uint32_t>(32 * (warp & 3)) << 16;
    const uint32_t o_addr = tmem_base + 256 + x * 128 + lane_field;
    AtRing vr;                          // V ring position of the unit's first key tile
    auto skip_v = [&](const ApUnit& w) { if (WIN) for (int j = 0; j < w.ntiles + (w.cut >= 0 ? 1 : 0); ++j) vr.advance(P::kVStages); };
    uint32_t s_phase = 0 /* bit per buffer */, o_phase = 0, q_phase = 0, done_phase = 0;      // done: of the last P V
    bool ok = true;
    // where there is one tile per unit, the next unit is looked up under the last products; with two it would cost registers
    ApUnit next = ap_unit<WIN, DEAL>(a, deal, list, 0);
    for (int wave = 0; wave < waves && ok; ++wave) {
      const ApUnit w = DEAL ? ap_unit<WIN, DEAL>(a, deal, list, wave) : next;
      const ApTile t = x == 0 ? w.t[0] : w.t[1];
      if (w.ntiles == 0 || !t.valid) {
        if (w.ntiles > 0) {
          if (!WIN && DEAL) {
            // a phase must have been seen complete before the next one can be waited for by parity
            ok = mbar_wait(bar(kApBarQFull), q_phase);
            if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
            if (lane == 0) mbar_arrive(bar(kApBarQReady + x));
          }
          q_phase ^= 1;
          skip_v(w);
        }
        if (!DEAL) next = ap_unit<WIN, DEAL>(a, deal, list, wave + 1);
        continue;
      }
      const int head = w.kvh * group + head_in_group;
      const int qi = t.m0 + tok_local, i = w.q_off + qi;
      const bool row_valid = row < rows_used && qi < w.Tq;
      const int S = 1 << a.log2_stairs;
      const int pad = ((w.T + S - 1) >> a.log2_stairs << a.log2_stairs) - w.T;
      // last (window form: and first) key this row sees
      const int limit = row_valid ? min(w.T - 1, ((((i + pad) >> a.log2_stairs) + 1) << a.log2_stairs) - 1 - pad) : -1;
      const int first = WIN && a.window > 0 ? i - a.window + 1 : 0;
      bf16* out_row = a.out + static_cast<int64_t>(w.q_start + (row_valid ? qi : 0)) * a.out_stride + head * (WIN ? a.dim : kHeadDim);
      if (!WIN) {
        // q * log2(e)/sqrt(D) rounded to bf16, in place (elementwise, so the swizzle does not matter)
        ok = mbar_wait(bar(kApBarQFull), q_phase);
        if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
        if (row < rows_used) {
          const uint32_t q_row = base + x * P::kQBytes + row * 128;
#pragma unroll
          for (int c = 0; c < 16; ++c) {
            const uint32_t addr = q_row + (c >> 3) * (128 * 128) + (c & 7) * 16;
            uint32_t z[4];
            asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(z[0]), "=r"(z[1]), "=r"(z[2]), "=r"(z[3]) : "r"(addr));
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float2 f = unpack_bf16x2(z[e]);
              z[e] = pack_bf16x2(f.x * a.q_scale, f.y * a.q_scale);
            }
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(z[0]), "r"(z[1]), "r"(z[2]), "r"(z[3]) : "memory");
          }
        }
        fence_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(kApBarQReady + x));
      }
      q_phase ^= 1;
      float m_ref = -INFINITY, l = 0.f;
      for (int j = t.first; j < t.last; ++j) {
        const int buf = !w.t[1].valid && (j & 1) ? kApAlone : x;
        const uint32_t s_addr = tmem_base + ap_score_col(buf) + lane_field;
        ok = mbar_wait(bar(kApBarSFull + buf), s_phase >> buf & 1);
        if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
        s_phase ^= 1u << buf;
        tc_fence_after();
        const int key0 = w.kbeg + j * kAtKeys;
        float s[kAtKeys];
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld32(s_addr + 32 * c, s + 32 * c);
        tmem_ld_wait();
        const int nv = limit + 1 - key0;            // keys of this tile the row sees: [0, nv)
        if (nv < kAtKeys) {
#pragma unroll
          for (int c = 0; c < kAtKeys; ++c) if (c >= nv) s[c] = -INFINITY;   // also replaces NaN from stale rows
        }
        if (WIN && first > key0) {
#pragma unroll
          for (int c = 0; c < kAtKeys; ++c) if (c < first - key0) s[c] = -INFINITY;
        }
        float mxv[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) mxv[k] = s[k];
#pragma unroll
        for (int c = 8; c < kAtKeys; c += 8) {
#pragma unroll
          for (int k = 0; k < 8; ++k) mxv[k] = fmaxf(mxv[k], s[c + k]);
        }
        float mx = fmaxf(fmaxf(fmaxf(mxv[0], mxv[1]), fmaxf(mxv[2], mxv[3])), fmaxf(fmaxf(mxv[4], mxv[5]), fmaxf(mxv[6], mxv[7])));
        if (!row_valid) mx = 0.f;                             // rows past the portion hold whatever the tile held
        const float m_tile = mx * a.scale_log2;
        // a row that sees no key of this tile (above the diagonal) keeps its state
        const bool grow = m_tile > m_ref + kAtRescaleStep || (m_ref == -INFINITY && m_tile != -INFINITY);
        if (__any_sync(0xffffffffu, grow)) {
          const float m_new = fmaxf(m_ref, m_tile);
          const float f = m_ref == -INFINITY ? 0.f : ex2_approx(m_ref - m_new);
          l *= f;
          if (j > t.first) {
            // O is quiet once the last key tile's P V has completed (the one before completed before these scores)
            ok = mbar_wait(bar(kApBarPDone + x), done_phase ^ 1);
            if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
            tc_fence_after();
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {
              float o[32];
              tmem_ld32(o_addr + 32 * c, o);
              tmem_ld_wait();
#pragma unroll
              for (int e = 0; e < 32; ++e) o[e] *= f;
              tmem_st32(o_addr + 32 * c, o);
            }
          }
          m_ref = m_new;
        }
        // P = 2^(s * scale - m_ref) rounded to bf16; a masked key gives 2^-inf = 0
        const float m_use = m_ref == -INFINITY ? 0.f : m_ref;   // nothing seen yet: every s is -inf, P = 0
        float lv[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float pk[32];                                         // 64 keys, two per word
#pragma unroll
          for (int c = 0; c < 64; c += 8) {
            float pv[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) pv[k] = ex2_approx(fmaf(s[64 * h + c + k], a.scale_log2, -m_use));
#pragma unroll
            for (int k = 0; k < 8; ++k) lv[k] += pv[k];
#pragma unroll
            for (int k = 0; k < 8; k += 2) pk[(c + k) >> 1] = __uint_as_float(pack_bf16x2(pv[k], pv[k + 1]));
          }
          tmem_st32(s_addr + 32 * h, pk);
        }
        l += ((lv[0] + lv[1]) + (lv[2] + lv[3])) + ((lv[4] + lv[5]) + (lv[6] + lv[7]));
        if (WIN && t.end - key0 < kAtKeys) {
          // values behind the tile's last key (stale cache rows, or tokens that only tile B sees) must not reach O through
          // 0 * (Inf or NaN): clear them.  Where A's keys end and B's go on, each has a copy of its own.
          AtRing v = vr;
          for (int n = 0; n < j + (x == 1 && w.cut >= 0 ? 1 : 0); ++n) v.advance(P::kVStages);
          ok = mbar_wait(bar(kApBarVFull + v.stage), v.phase);
          if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
          const uint32_t v_tile = base + P::kOffV + v.stage * kAtTileBytes;
          const int r = t.end - key0 + row;
          if (r < kAtKeys) {
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
              for (int c = 0; c < 8; ++c)
                asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(v_tile + h * kAtHalfBytes + r * 128 + c * 16),
                             "r"(0u)
                             : "memory");
          }
          fence_async_smem();
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(kApBarPFull + buf));
        done_phase ^= 1;
      }
      if (!ok) break;
      skip_v(w);
      if (!DEAL) next = ap_unit<WIN, DEAL>(a, deal, list, wave + 1);
      // ------------------------------------------------------------- outputs of the tile
      ok = mbar_wait(bar(kApBarOFull + x), o_phase);
      if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
      o_phase ^= 1;
      tc_fence_after();
      float inv;
      if (WIN) {
        // the sink's term exp(0) in the units of the running reference
        const float den = a.sink ? l + ex2_approx(-m_ref) : l;
        float z = a.out_scale;
        if (row_valid && rows_present(a.gate)) z *= sigmoid_f(rows_at<bf16>(a.gate, w.q_start + t.m0 + tok_local, head));
        inv = den > 0.f ? z / den : 0.f;
      } else {
        inv = l > 0.f ? 1.0f / l : 0.f;
      }
      const bool ragged = WIN && a.dim != 64 * halves;      // fewer channels leave than are stored
#pragma unroll 1
      for (int c = 0; c < 2 * halves; ++c) {
        float o[32];
        tmem_ld32(o_addr + 32 * c, o);
        tmem_ld_wait();
        if (row_valid && ragged) {
#pragma unroll
          for (int e = 0; e < 32; ++e)
            if (32 * c + e < a.dim) out_row[32 * c + e] = __float2bfloat16_rn(o[e] * inv);
        } else if (row_valid) {
#pragma unroll
          for (int q4 = 0; q4 < 4; ++q4)
            reinterpret_cast<uint4*>(out_row + 32 * c)[q4] =
                make_uint4(pack_bf16x2(o[8 * q4] * inv, o[8 * q4 + 1] * inv), pack_bf16x2(o[8 * q4 + 2] * inv, o[8 * q4 + 3] * inv),
                           pack_bf16x2(o[8 * q4 + 4] * inv, o[8 * q4 + 5] * inv), pack_bf16x2(o[8 * q4 + 6] * inv, o[8 * q4 + 7] * inv));
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(kApBarOEmpty + x));
    }
    if (!ok && lane == 0) report_status(MDB_STATUS_WAIT_TIMEOUT);
  }

  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

template <bool WIN, bool DEAL>
static int ap_run(const CUtensorMap& map_q, const CUtensorMap& map_k, const CUtensorMap& map_v, const AtArgs& a, int units, int grid, cudaStream_t st) {
  static PerDeviceOnce attr_once;
  const int dev = attr_once.slot();
  if (dev < 0) return MDB_ERR_CUDA;
  if (!attr_once.done[dev]) {
    if (cudaFuncSetAttribute(attn_prompt_kernel<WIN, DEAL>, cudaFuncAttributeMaxDynamicSharedMemorySize, ApPlan::kSmemBytes) != cudaSuccess)
      return MDB_ERR_CUDA;
    attr_once.done[dev] = true;
  }
  return mdb_launch(attn_prompt_kernel<WIN, DEAL>, dim3(grid), dim3(ApRoles<DEAL>::kThreads), ApPlan::kSmemBytes, st, map_q, map_k, map_v, a, units);
}

// Tiles per unit for sequences of the same `queries` and `keys` (each of the first behind keys - queries tokens): the shorter time of
// the longest of every fourth CTA.  One prompt of 1280 to 2304 tokens (160 to 288 tiles): 31 - 49 us in pairs, 19 - 35 us alone; of 4096
// tokens, or 8 of 256, the other way round (79 against 84, 17 against 19 us).
template <bool WIN>
static int ap_tiles_alike(const AtArgs& a, int queries, int keys, int sms) {
  const int per_rank = a.nseq * a.hkv;
  if (a.max_qtiles == 1) return 1;
  if (static_cast<int64_t>(a.max_qtiles) * per_rank > 4 * sms) return 2;
  const ApSeq w = {0, queries, keys - queries, keys, 0};
  int most[2] = {0, 0};
  for (int per = 1; per <= 2; ++per) {
    const int n = (a.max_qtiles + per - 1) / per;
    for (int c = 0; c < sms; c += 4) {
      int t = 0;
      for (int p0 = 0, odd = 0; p0 < n * per_rank; p0 += sms, odd ^= 1) {
        const int p = p0 + (odd ? sms - 1 - c : c);
        if (p < n * per_rank) t += ap_cost<WIN>(a, w, (n - 1 - p / per_rank) * per, per == 2);
      }
      if (t > most[per - 1]) most[per - 1] = t;
    }
  }
  // (a launch of tiles alone, with 192 threads, takes 0.87 of the time of one that could have had pairs: 30.5 against 35.1 us for 2048)
  return 7 * most[0] <= 8 * most[1] ? 1 : 2;
}

// Tiles that can all have an SM of their own take one: two on one SM wait for one another (one prompt of 1056 tokens, 136 tiles:
// 24.8 us in pairs, 19.0 us alone).  With more, a.tiles_per_unit is the answer for sequences that are alike, or 0: the kernel decides.
template <bool WIN>
static int ap_launch(const CUtensorMap& map_q, const CUtensorMap& map_k, const CUtensorMap& map_v, const AtArgs& a, cudaStream_t st) {
  const int sms = at_sm_count();
  const int64_t tiles = static_cast<int64_t>(a.max_qtiles) * a.nseq * a.hkv;
  if (tiles > (1 << 30)) return MDB_ERR_UNSUPPORTED;
  const int units = static_cast<int>(tiles), grid = units < sms ? units : sms;
  return units <= sms || a.tiles_per_unit == 1 ? ap_run<WIN, false>(map_q, map_k, map_v, a, units, grid, st)
                                               : ap_run<WIN, true>(map_q, map_k, map_v, a, units, grid, st);
}

// ---- staircase form ----
static bool attn_stair_tc_supported(int hq, int hkv, int64_t q_stride, int64_t k_stride, int64_t v_stride) {
  if (hkv <= 0 || hq % hkv != 0 || hq / hkv > 128) return false;
  return q_stride % 8 == 0 && k_stride % 8 == 0 && v_stride % 8 == 0;
}

static int attn_stair_tc_launch(const AttnStairArgs& sa, int nseq, int max_seqlen, int64_t total_q, int64_t total_tokens,
                                cudaStream_t st) {
  AtArgs a = {};
  a.q = sa.q;
  a.out = sa.out;
  a.hq = sa.hq; a.hkv = sa.hkv; a.group = sa.hq / sa.hkv;
  a.scale_log2 = sa.scale_log2;
  a.q_scale = sa.q_scale;
  a.cu_seqlens = sa.cu_seqlens;
  a.cu_seqlens_q = sa.cu_seqlens_q;
  a.out_stride = sa.out_stride;
  a.nseq = nseq;
  a.log2_stairs = sa.log2_stairs;
  a.tokens_per_unit = 128 / a.group;
  a.max_qtiles = (max_seqlen + a.tokens_per_unit - 1) / a.tokens_per_unit;
  // one sequence, or prompts of one length (an odd last tile would be first in the order, and not the longest unit); one tile each
  if (a.max_qtiles == 1 || (nseq == 1 && total_q == max_seqlen && total_tokens >= total_q) ||
      (a.max_qtiles % 2 == 0 && total_q == static_cast<int64_t>(nseq) * max_seqlen && total_q == total_tokens))
    a.tiles_per_unit = ap_tiles_alike<false>(a, max_seqlen, nseq == 1 ? static_cast<int>(total_tokens) : max_seqlen, at_sm_count());
  a.nsplit = 1;
  CUtensorMap map_q, map_k, map_v;
  if (!get_q_tensor_map(sa.q, total_q, sa.q_stride, sa.hq, a.group, a.tokens_per_unit, &map_q)) return MDB_ERR_CUDA;
  if (!get_tensor_map(sa.k, total_tokens, sa.hkv * kHeadDim, sa.k_stride, kAtKeys, &map_k)) return MDB_ERR_CUDA;
  if (!get_tensor_map(sa.v, total_tokens, sa.hkv * kHeadDim, sa.v_stride, kAtKeys, &map_v)) return MDB_ERR_CUDA;
  return ap_launch<false>(map_q, map_k, map_v, a, st);
}

// ---- window form ----
static bool attn_win_tc_supported(const mdb_window_attn_args& w) {
  return w.dtype == MDB_BF16 && (w.dim_pad == 64 || w.dim_pad == 128) && w.heads / w.kv_heads <= 128 && w.scale > 0.f && w.cu_q && w.start;
}

static int attn_win_tc_launch(const mdb_window_attn_args& w, cudaStream_t st) {
  AtArgs a = {};
  a.q = static_cast<const bf16*>(w.q);
  a.out = static_cast<bf16*>(w.out);
  a.hq = w.heads; a.hkv = w.kv_heads; a.group = w.heads / w.kv_heads;
  a.scale_log2 = w.scale * 1.4426950408889634f;
  a.q_scale = 1.0f;
  a.cu_seqlens_q = w.cu_q;
  a.start = w.start;
  a.block_table = w.block_table;
  a.table_stride = w.table_stride;
  a.num_pages = w.num_pages;
  a.out_stride = w.ld_out;
  a.nseq = w.bs;
  a.tokens_per_unit = 128 / a.group;
  a.max_qtiles = (w.max_q + a.tokens_per_unit - 1) / a.tokens_per_unit;
  // one tile each; portions of one length under a narrow window, which makes their tiles alike, wherever they start
  if (a.max_qtiles == 1 || (a.max_qtiles % 2 == 0 && w.m == static_cast<int64_t>(w.bs) * w.max_q && w.window > 0 && w.window <= 2 * kAtKeys))
    a.tiles_per_unit = ap_tiles_alike<true>(a, w.max_q, w.max_q + w.window, at_sm_count());
  a.nsplit = 1;
  a.window = w.window; a.sink = w.sink;
  a.dim = w.dim; a.halves = w.dim_pad / 64;
  a.out_scale = w.out_scale;
  a.gate = w.gate;
  CUtensorMap map_q, map_k, map_v;
  const int64_t cache_rows = static_cast<int64_t>(w.num_pages) * kPage;
  const int cols = w.kv_heads * w.dim_pad;
  if (!get_q_tensor_map(w.q, w.m, static_cast<int64_t>(w.heads) * w.dim_pad, w.heads, a.group, a.tokens_per_unit, &map_q, w.dim_pad)) return MDB_ERR_CUDA;
  if (!get_tensor_map(w.k_cache, cache_rows, cols, cols, kAtKeys, &map_k)) return MDB_ERR_CUDA;
  if (!get_tensor_map(w.v_cache, cache_rows, cols, cols, kAtKeys, &map_v)) return MDB_ERR_CUDA;
  return ap_launch<true>(map_q, map_k, map_v, a, st);
}

}  // namespace mdb
