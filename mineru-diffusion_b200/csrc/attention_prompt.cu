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
// 4 x 4096 tokens, 16 query and 8 KV heads: 400 -> 301 us alone, 417 -> 335 in a loop at the power limit, the same bits.  (Steps of
// 64 keys with two score buffers per tile and an issuing warp per tile: 299 us alone, 329 in a loop, other roundings; an issuing
// warp per tile with these steps: 351.)
//
// Tensor memory: S_A (P_A) | S_B (P_B) | O_A | O_B, 128 columns each; with one tile S of even | odd key tiles | O.
#include "mdb_common.cuh"

namespace mdb {

struct ApPlan {
  static constexpr int kKStages = 3, kVStages = 2;
  static constexpr int kQBytes = 2 * 128 * 128;             // a tile: two channel halves of [128 rows][128 B]
  static constexpr int kProducerWarp = 8, kMmaWarp = 9, kThreads = 384;      // three warpgroups; two warps idle
  // registers: 384 threads x 168 at launch = 256 x 216 (softmax) + 128 x 72
  static constexpr int kSoftmaxRegs = 216, kOtherRegs = 72;
  static_assert(256 * kSoftmaxRegs + 128 * kOtherRegs <= kThreads * 168, "registers after the split");
  static constexpr int kOffK = 2 * kQBytes;
  static constexpr int kOffV = kOffK + kKStages * kAtTileBytes;
  static constexpr int kOffBars = kOffV + kVStages * kAtTileBytes;
  static constexpr int kSmemBytes = 1024 + kOffBars + 256;
};
static_assert(ApPlan::kSmemBytes <= 227 * 1024, "shared memory of the prompt attention");

// barrier slots; those of a tile (A, B) or of a score buffer come in pairs
enum {
  kApBarQFull = 0, kApBarQEmpty = 1, kApBarQReady = 2, kApBarKFull = 4, kApBarKEmpty = 7, kApBarVFull = 10, kApBarVEmpty = 12,
  kApBarSFull = 14, kApBarPFull = 16, kApBarPDone = 18, kApBarOFull = 20, kApBarOEmpty = 22, kApBarCount = 24
};

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

// Units are (pair of query tiles, sequence, KV head), the late (long) pairs first, dealt to the CTAs in alternating direction;
// with tiles_per_unit 1 there is no tile B.
template <bool WIN>
__device__ __forceinline__ ApUnit ap_unit(const AtArgs& a, int units, int wave) {
  ApUnit w = {};
  w.cut = -1;
  const int G = static_cast<int>(gridDim.x), c = static_cast<int>(blockIdx.x);
  const int p = wave * G + ((wave & 1) ? G - 1 - c : c);
  if (p >= units) return w;
  const int per_pair = a.nseq * a.hkv, pairs = (a.max_qtiles + a.tiles_per_unit - 1) / a.tiles_per_unit;
  const int pair = pairs - 1 - p / per_pair, rest = p % per_pair;
  w.seq = rest / a.hkv;
  w.kvh = rest % a.hkv;
  const int32_t* cu_q = a.cu_seqlens_q != nullptr ? a.cu_seqlens_q : a.cu_seqlens;
  w.q_start = cu_q[w.seq];
  w.Tq = cu_q[w.seq + 1] - w.q_start;
  if (WIN) {
    w.q_off = a.start[w.seq];
    w.T = w.q_off + w.Tq;
  } else {
    w.seq_start = a.cu_seqlens[w.seq];
    w.T = a.cu_seqlens[w.seq + 1] - w.seq_start;
    w.q_off = w.T - w.Tq;
  }
  const int S = 1 << a.log2_stairs;
  const int pad = ((w.T + S - 1) >> a.log2_stairs << a.log2_stairs) - w.T;
#pragma unroll
  for (int x = 0; x < 2; ++x) {
    ApTile& t = w.t[x];
    t.m0 = (a.tiles_per_unit * pair + x) * a.tokens_per_unit;
    t.valid = x < a.tiles_per_unit && t.m0 < w.Tq;
    if (!t.valid) continue;
    const int last = w.q_off + min(t.m0 + a.tokens_per_unit, w.Tq) - 1;
    const int end = min(w.T, ((((last + pad) >> a.log2_stairs) + 1) << a.log2_stairs) - pad);
    // window form: from the tile of keys that holds the first query's first key
    const int beg = WIN && a.window > 0 ? max(0, w.q_off + t.m0 - a.window + 1) : 0;
    if (x == 0) w.kbeg = beg / kAtKeys * kAtKeys;
    t.end = end;
    t.first = (beg - w.kbeg) / kAtKeys;
    t.last = (end - w.kbeg + kAtKeys - 1) / kAtKeys;
    w.ntiles = t.last;
  }
  if (WIN && w.t[1].valid && w.t[0].end < w.kbeg + w.t[0].last * kAtKeys) w.cut = w.t[0].last - 1;
  return w;
}

template <bool WIN>
__global__ void __launch_bounds__(ApPlan::kThreads, 1)
attn_prompt_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                   const __grid_constant__ CUtensorMap map_v, const AtArgs a, const int units) {
  using P = ApPlan;
  const int halves = WIN ? a.halves : 2;      // 64-channel halves of a stored head
  extern __shared__ __align__(1024) unsigned char ap_smem_raw[];
  const uint32_t raw = smem_u32(ap_smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  unsigned char* gen_base = ap_smem_raw + (base - raw);
  const uint32_t bars = base + P::kOffBars;
  auto bar = [&](int slot) { return bars + 8u * static_cast<uint32_t>(slot); };
  volatile uint32_t* misc = reinterpret_cast<volatile uint32_t*>(gen_base + P::kOffBars + 8 * kApBarCount);
  const int waves = (units + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int group = a.group;
  const int rows_used = group * a.tokens_per_unit;      // <= 128

  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    for (int s = 0; s < kApBarCount; ++s) {
      const bool by_softmax = s == kApBarQReady || s == kApBarQReady + 1 || (s >= kApBarPFull && s < kApBarPFull + 2) || s >= kApBarOEmpty;
      mbar_init(bar(s), by_softmax ? 4 : 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == P::kMmaWarp) {
    const uint32_t slot = smem_u32(const_cast<uint32_t*>(&misc[0]));
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = misc[0];
  pdl_wait();   // q and the K/V rows of this step come from the preceding kernels

  if (warp >= P::kProducerWarp) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(P::kOtherRegs));
    if (warp == P::kProducerWarp) {
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
          const ApUnit w = ap_unit<WIN>(a, units, wave);
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
    } else if (warp == P::kMmaWarp) {
      // ----------------------------------------------------------------- MMA issue (all lanes, one elected)
      const bool single = a.tiles_per_unit == 1;
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
        const ApUnit w = ap_unit<WIN>(a, units, wave);
        if (w.ntiles == 0) continue;
        if (WIN) {
          if (!mbar_wait_w(bar(kApBarQFull), qfull_phase)) { ok = false; break; }
          qfull_phase ^= 1;
        } else {
          // staircase form: the softmax warps scale q in place first.  Those of a tile that is not there have only seen it: the
          // next unit's q may not arrive before all have, or they would miss a phase and wait for a later one.
          if (!mbar_wait_w(bar(kApBarQReady), qfull_phase) || !mbar_wait_w(bar(kApBarQReady + 1), qfull_phase)) { ok = false; break; }
          qfull_phase ^= 1;
        }
        auto issue_s = [&](int x, int buf) {           // scores of tile x with the K tile at the ring's position
          const uint32_t q_tile = base + x * P::kQBytes, k_tile = base + P::kOffK + kr.stage * kAtTileBytes;
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            if (WIN && c >= halves) break;
            umma_bf16_x4_w(tmem_base + buf * 128, umma_desc_sw128(q_tile + c * (128 * 128)), 2, umma_desc_sw128(k_tile + c * kAtHalfBytes), 2,
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
          if (single && more) {
            // the other buffer held the last key tile, whose P V has been issued
            if (!mbar_wait_w(bar(kApBarKFull + kr.stage), kr.phase)) { ok = false; break; }
            tc_fence_after();
            issue_s(0, (j + 1) & 1);
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
              const int buf = single ? j & 1 : x;
              if (j == w.t[x].first) {
                // the previous unit's accumulator must have been read out
                if (!mbar_wait_w(bar(kApBarOEmpty + x), o_phase[x] ^ 1)) { ok = false; break; }
                o_phase[x] ^= 1;
              }
              if (!mbar_wait_w(bar(kApBarPFull + buf), p_phase >> buf & 1)) { ok = false; break; }
              p_phase ^= 1u << buf;
              tc_fence_after();
              const uint32_t v_tile = base + P::kOffV + vr.stage * kAtTileBytes, p = tmem_base + buf * 128, o = tmem_base + 256 + x * 128;
              umma_bf16_ts_x4_w(o, p, umma_desc_sw128_mn(v_tile), 128, idesc_o, j > w.t[x].first ? 1u : 0u);
              umma_bf16_ts_x4_w(o, p + 32, umma_desc_sw128_mn(v_tile + 4 * 2048), 128, idesc_o, 1u);
              umma_commit_w(bar(kApBarPDone + x));
              if (j == w.t[x].last - 1) umma_commit_w(bar(kApBarOFull + x));
            }
            if (!single && more && j + 1 >= w.t[x].first && j + 1 < w.t[x].last) {
              if (!k_there && !mbar_wait_w(bar(kApBarKFull + kr.stage), kr.phase)) { ok = false; break; }
              k_there = true;
              tc_fence_after();
              issue_s(x, x);
            }
          }
          if (!ok) break;
          umma_commit_w(bar(kApBarVEmpty + vr.stage));
          vr.advance(P::kVStages);
          if (!single && more) release_k(j + 1);      // (the key tiles of A and B overlap or touch: every one is used by a tile)
        }
      }
      if (!ok && lane == 0) report_status(MDB_STATUS_WAIT_TIMEOUT);
    }
  } else {
    // ------------------------------------------------------------------- softmax
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(P::kSoftmaxRegs));
    const int x = warp >> 2;                               // tile A or B
    const int row = threadIdx.x & 127;                     // query row of the tile, and its tensor-memory lane
    const int tok_local = row / group, head_in_group = row % group;
    const uint32_t lane_field = static_cast<uint32_t>(32 * (warp & 3)) << 16;
    const bool single = a.tiles_per_unit == 1;
    const uint32_t o_addr = tmem_base + 256 + x * 128 + lane_field;
    AtRing vr;                          // V ring position of the unit's first key tile
    auto skip_v = [&](const ApUnit& w) { if (WIN) for (int j = 0; j < w.ntiles + (w.cut >= 0 ? 1 : 0); ++j) vr.advance(P::kVStages); };
    uint32_t s_phase = 0 /* bit per buffer */, o_phase = 0, q_phase = 0, done_phase = 0;      // done: of the last P V
    bool ok = true;
    for (int wave = 0; wave < waves && ok; ++wave) {
      const ApUnit w = ap_unit<WIN>(a, units, wave);
      if (w.ntiles == 0) continue;
      const ApTile t = x == 0 ? w.t[0] : w.t[1];
      if (!t.valid) {
        if (!WIN) {
          // a phase must have been seen complete before the next one can be waited for by parity
          ok = mbar_wait(bar(kApBarQFull), q_phase);
          if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
          if (lane == 0) mbar_arrive(bar(kApBarQReady + x));
        }
        q_phase ^= 1;
        skip_v(w);
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
        const int buf = single ? j & 1 : x;
        const uint32_t s_addr = tmem_base + buf * 128 + lane_field;
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
  if (warp == P::kMmaWarp) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

template <bool WIN>
static int ap_launch(const CUtensorMap& map_q, const CUtensorMap& map_k, const CUtensorMap& map_v, AtArgs& a, cudaStream_t st) {
  static PerDeviceOnce attr_once;
  const int dev = attr_once.slot();
  if (dev < 0) return MDB_ERR_CUDA;
  if (!attr_once.done[dev]) {
    if (cudaFuncSetAttribute(attn_prompt_kernel<WIN>, cudaFuncAttributeMaxDynamicSharedMemorySize, ApPlan::kSmemBytes) != cudaSuccess)
      return MDB_ERR_CUDA;
    attr_once.done[dev] = true;
  }
  // Tiles that can all have an SM of their own take one: two on one SM wait for one another (one prompt of 1056
  // tokens, 136 tiles: 24.8 us in pairs, 20.4 us alone).
  const int sms = at_sm_count();
  a.tiles_per_unit = static_cast<int64_t>(a.max_qtiles) * a.nseq * a.hkv <= sms ? 1 : 2;
  const int64_t units = static_cast<int64_t>((a.max_qtiles + a.tiles_per_unit - 1) / a.tiles_per_unit) * a.nseq * a.hkv;
  if (units > (1 << 30)) return MDB_ERR_UNSUPPORTED;
  const int grid = units < sms ? static_cast<int>(units) : sms;
  return mdb_launch(attn_prompt_kernel<WIN>, dim3(grid), dim3(ApPlan::kThreads), ApPlan::kSmemBytes, st, map_q, map_k, map_v, a,
                    static_cast<int>(units));
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
