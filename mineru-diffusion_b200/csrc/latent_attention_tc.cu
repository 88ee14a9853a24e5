// Causal attention over cached latents on the 5th-generation tensor cores (bf16, widths of 128 to 512): every query head of a
// token reads the same latent row of a key, which stands for its key and its value alike.
//
// Both products are turned so that the long sides fill the matrix unit and the heads are its narrow side:
//   S^T [64 keys x heads]      = C Q^T        (C the tile of 64 latents, K-major; M = 64, N = 16 or 32 heads)
//   O^T [width x 2 x heads]   += C^T P^T      (C once more, M-major; M = 128 channels, N = high and low parts of P)
// The weights enter as the sum of two bf16 numbers side by side, so they keep 16 significant bits.  Roles: a TMA warp (a ring
// of latent tiles, boxes of 64 keys x 64 channels), an MMA warp, four softmax warps.  S^T has keys in the lanes, so it is
// turned around in shared memory; eight threads then share a head.  O^T is rescaled only when a head's maximum has grown
// by more than 2^8.
//
// What bounds it: memory; a tile is read from shared memory twice (1024 cycles at 64 KB) and written once.  A CTA per SM takes
// an equal share of all the step's key tiles, cut where they fall (a row of a step has at most nsplit parts; with one part
// rows stay whole), so with three parts a row and more a ragged batch leaves no SM behind; with two a share is at least the longest
// row, and 99 to 148 rows keep as many SMs busy.  The next row's tiles arrive while this one's output leaves.
// With the merge of the parts, 16 heads, width 512: 32 requests of 2048 to 4096 keys 47.3 -> 31.7 us, 60 requests 79.9 -> 46.1,
// one request of 8000 keys 32.2 -> 28.4, of 300 keys 17.9 -> 18.1; 64 requests of 4000 to 8000 keys, 32 heads, 263 -> 169 us.
#include "mdb_common.cuh"

namespace mdb {

constexpr int kLtKeys = 64, kLtThreads = 192, kLtBox = kLtKeys * 128;      // bytes of a box of 64 channels

template <int WIDTH, int HG>
struct LtPlan {
  static constexpr int NB = WIDTH / 64, NM = WIDTH / 128, HEADS = 16 * HG;
  static constexpr int kStage = NB * kLtBox;
  static constexpr int kStages = WIDTH > 384 ? (HG == 1 ? 3 : 2) : WIDTH > 256 ? 3 : 4;
  static constexpr int kQBytes = NB * HEADS * 128, kPBytes = 2 * HEADS * 128;
  static constexpr int kSLd = kLtKeys + 4;                                  // floats between the heads of a turned tile
  static constexpr int kOffQ = kStages * kStage, kOffP = kOffQ + kQBytes, kOffS = kOffP + 2 * kPBytes;
  static constexpr int kOffF = kOffS + 2 * HEADS * kSLd * 4, kOffBars = kOffF + HEADS * 4, kBytes = 1024 + kOffBars + 8 * 32 + 64;
  static constexpr uint32_t kTmemO = 2 * HEADS;                             // columns: S, S, O of each 128 channels
  static_assert(kBytes <= 227 * 1024, "shared memory of the latent attention");
  static_assert(kTmemO + NM * 2 * HEADS <= 512, "tensor memory of the latent attention");
};
enum { kLtBarKFull = 0, kLtBarKEmpty = 4, kLtBarQFull = 8, kLtBarQEmpty, kLtBarSFull, kLtBarSEmpty = kLtBarSFull + 2, kLtBarPFull = kLtBarSEmpty + 2,
       kLtBarPEmpty = kLtBarPFull + 2, kLtBarOFull = kLtBarPEmpty + 2, kLtBarOEmpty, kLtBarCount };
static_assert(8 * kLtBarCount + 8 <= 8 * 32, "barriers of the latent attention");

// C^T as the left operand: channels (64 per 128-byte row, the next 64 one box on) by keys (rows, groups of eight 1024 bytes apart)
__device__ __forceinline__ uint64_t lt_desc_mn(uint32_t smem_addr) {
  return static_cast<uint64_t>((smem_addr >> 4) & 0x3FFF) | (static_cast<uint64_t>(kLtBox >> 4) << 16) | (static_cast<uint64_t>(1024 >> 4) << 32) |
         (static_cast<uint64_t>(1) << 46) | (static_cast<uint64_t>(2) << 61);
}

// The share of a CTA: `count` key tiles of the rows laid end to end, from tile `off` of row `row`, which begins at `base`.
struct LtShare {
  int row, off, count, base, per_cta;
};
// Walks the parts of rows in a share.
struct LtPart {
  int row, keys, tile0, tiles, part, parts;
};
struct LtWalk {
  LtShare s;
  bool whole;
  __device__ __forceinline__ bool next(const LatentArgs& a, LtPart& p) {
    for (; s.count > 0 && s.row < a.m; ++s.row) {
      const int keys = max(0, a.row_pos[s.row] + 1), n = (keys + kLtKeys - 1) / kLtKeys;
      if (n == 0) continue;
      p.row = s.row;
      p.keys = keys;
      p.tile0 = s.off;
      p.tiles = whole ? n : min(n - s.off, s.count);
      const int first = s.base / s.per_cta;
      p.part = whole ? 0 : (s.base + s.off) / s.per_cta - first;
      p.parts = whole ? 1 : (s.base + n - 1) / s.per_cta - first + 1;
      s.count -= p.tiles;
      s.off += p.tiles;
      if (s.off >= n) { s.base += n; s.off = 0; ++s.row; }
      return true;
    }
    return false;
  }
};

// Every CTA's share of the rows' key tiles, by one warp: equal counts of the rows laid end to end, where no row may be cut into
// more than nsplit parts.  That allows for a cut inside a part, so with few parts per row (2 for 5 rows of 300 keys) the
// shares grow long: where there are CTAs for all parts and the shares get no shorter, rows are cut into nsplit equal parts instead.
__device__ __forceinline__ LtShare lt_share(const LatentArgs& a, int cta, int ctas, int lane) {
  auto tiles_of = [&](int r) { return r < a.m ? (max(0, a.row_pos[r] + 1) + kLtKeys - 1) / kLtKeys : 0; };
  const int n_first = tiles_of(lane);
  int total = n_first, most = n_first;
  for (int r = lane + 32; r < a.m; r += 32) {
    const int n = tiles_of(r);
    total += n;
    most = max(most, n);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    total += __shfl_xor_sync(0xffffffffu, total, o);
    most = max(most, __shfl_xor_sync(0xffffffffu, most, o));
  }
  LtShare s = {};
  s.per_cta = max(1, (total + ctas - 1) / ctas);
  if (a.nsplit > 1) {
    s.per_cta = max(s.per_cta, (most + a.nsplit - 2) / (a.nsplit - 1));
    if (static_cast<int64_t>(a.m) * a.nsplit <= ctas && (most + a.nsplit - 1) / a.nsplit <= s.per_cta) {
      s.row = cta / a.nsplit;
      const int n = tiles_of(s.row);
      s.per_cta = max(1, (n + a.nsplit - 1) / a.nsplit);
      s.off = cta % a.nsplit * s.per_cta;
      s.count = max(0, min(s.per_cta, n - s.off));
      return s;
    }
  }
  const int begin = cta * s.per_cta, end = min(total, begin + s.per_cta);
  if (begin >= end) return s;
  // the row that holds tile `begin`; with whole rows, the first row that starts at or behind it
  int before = 0;
  for (int r0 = 0; r0 < a.m; r0 += 32) {
    const int r = r0 + lane;
    int n = r0 == 0 ? n_first : tiles_of(r);
    const int mine = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, n, o);
      if (lane >= o) n += up;
    }
    const int start = before + n - mine;
    const bool here = mine > 0 && (a.nsplit > 1 ? start <= begin && begin < start + mine : start >= begin && start < end);
    const uint32_t found = __ballot_sync(0xffffffffu, here);
    if (found) {
      const int src = __ffs(found) - 1;
      s.row = r0 + src;
      s.base = __shfl_sync(0xffffffffu, start, src);
      s.off = a.nsplit > 1 ? begin - s.base : 0;
      s.count = end - (a.nsplit > 1 ? begin : s.base);      // whole rows: as long as one starts inside
      return s;
    }
    before += __shfl_sync(0xffffffffu, n, 31);
  }
  return s;
}

template <int WIDTH, int HG>
__global__ void __launch_bounds__(kLtThreads, 1)
latent_attn_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_c, const LatentArgs a) {
  using P = LtPlan<WIDTH, HG>;
  constexpr int NB = P::NB, NM = P::NM, HEADS = P::HEADS;
  extern __shared__ __align__(1024) unsigned char lt_smem_raw[];
  const uint32_t raw = smem_u32(lt_smem_raw), base = (raw + 1023u) & ~1023u;
  unsigned char* mem = lt_smem_raw + (base - raw);
  const uint32_t bars = base + P::kOffBars;
  auto bar = [&](int slot) { return bars + 8u * static_cast<uint32_t>(slot); };
  volatile uint32_t* misc = reinterpret_cast<volatile uint32_t*>(mem + P::kOffBars + 8 * kLtBarCount);
  int* share = reinterpret_cast<int*>(mem + P::kOffBars + 8 * 32);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int groups = (a.heads + HEADS - 1) / HEADS, head0 = static_cast<int>(blockIdx.x) % groups * HEADS;
  const int nh = min(HEADS, a.heads - head0);

  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    misc[1] = 0;
    for (int s = 0; s < kLtBarCount; ++s) {
      const bool by_softmax = (s >= kLtBarSEmpty && s < kLtBarSEmpty + 2) || (s >= kLtBarPFull && s < kLtBarPFull + 2) || s == kLtBarOEmpty;
      mbar_init(bar(s), by_softmax ? 4 : 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 5) {
    const uint32_t slot = smem_u32(const_cast<uint32_t*>(&misc[0]));
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  pdl_wait();
  if (warp == 0) {
    const LtShare s = lt_share(a, static_cast<int>(blockIdx.x) / groups, static_cast<int>(gridDim.x) / groups, lane);
    if (lane == 0) { share[0] = s.row; share[1] = s.off; share[2] = s.count; share[3] = s.base; share[4] = s.per_cta; }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = misc[0];
  // A wait that runs out raises the abort flag; the softmax warps, who meet at barriers, then walk to the end without waiting.
  auto wait = [&](int slot, uint32_t parity) {
    uint32_t done;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(done) : "r"(bar(slot)), "r"(parity) : "memory");
    if (done || misc[1] != 0) return;
    if (!mbar_wait(bar(slot), parity)) {
      misc[1] = 1;
      report_status(MDB_STATUS_WAIT_TIMEOUT);
    }
  };
  LtWalk walk = {{share[0], share[1], share[2], share[3], share[4]}, a.nsplit == 1};
  LtPart w;

  if (warp == 4) {
    // ------------------------------------------------------------------ producer
    if (lane == 0) {
      AtRing kr;
      uint32_t q_phase = 0, pend_k = 0, par_k = 0, pend_q = 0;
      bool ok = true;
      while (ok && walk.next(a, w)) {
        if (!mbar_wait(bar(kLtBarQEmpty), q_phase ^ 1)) { ok = false; break; }
        mbar_arrive_expect_tx(bar(kLtBarQFull), P::kQBytes);
        for (int b = 0; b < NB; ++b) tma_load_2d(base + P::kOffQ + b * HEADS * 128, &map_q, b * 64, w.row * a.heads + head0, bar(kLtBarQFull));
        pend_q = 1;
        q_phase ^= 1;
        const int32_t* table = a.table + static_cast<int64_t>(a.row_seq[w.row]) * a.table_stride;
        for (int t = 0; t < w.tiles; ++t) {
          if (!mbar_wait(bar(kLtBarKEmpty + kr.stage), kr.phase ^ 1)) { ok = false; break; }
          const uint32_t full = bar(kLtBarKFull + kr.stage), dst = base + kr.stage * P::kStage;
          const int slot = static_cast<int>(latent_slot(a, table, (w.tile0 + t) * kLtKeys));
          mbar_arrive_expect_tx(full, P::kStage);
          for (int b = 0; b < NB; ++b) tma_load_2d(dst + b * kLtBox, &map_c, b * 64, slot, full);
          pend_k |= 1u << kr.stage;
          par_k = (par_k & ~(1u << kr.stage)) | (kr.phase << kr.stage);
          kr.advance(P::kStages);
        }
      }
      if (!ok) {
        misc[1] = 1;
        report_status(MDB_STATUS_WAIT_TIMEOUT);
        // let the copies already issued land before the CTA gives its shared memory back
        for (int s = 0; s < P::kStages; ++s) if (pend_k >> s & 1) mbar_wait(bar(kLtBarKFull + s), par_k >> s & 1);
        if (pend_q) mbar_wait(bar(kLtBarQFull), q_phase ^ 1);
      }
    }
  } else if (warp == 5) {
    // ----------------------------------------------------------------- MMA issue (all lanes, one elected)
    const uint32_t kBf16 = (1u << 4) | (1u << 7) | (1u << 10);               // bf16 x bf16 -> fp32
    const uint32_t idesc_s = kBf16 | (static_cast<uint32_t>(HEADS >> 3) << 17) | (static_cast<uint32_t>(64 >> 4) << 24);
    const uint32_t idesc_o = kBf16 | (1u << 15) | (static_cast<uint32_t>(2 * HEADS >> 3) << 17) | (static_cast<uint32_t>(128 >> 4) << 24);
    AtRing kr, ks, sr, pr;          // latent tile of the next O += C^T P^T and of the next S; S and P buffers
    uint32_t q_phase = 0, o_phase = 0;
    bool ok = true;
    while (ok && walk.next(a, w)) {
      if (!mbar_wait_w(bar(kLtBarQFull), q_phase)) { ok = false; break; }
      q_phase ^= 1;
      auto issue_s = [&](int t) {
        if (!mbar_wait_w(bar(kLtBarKFull + ks.stage), ks.phase)) return false;
        if (!mbar_wait_w(bar(kLtBarSEmpty + sr.stage), sr.phase ^ 1)) return false;
        tc_fence_after();
#pragma unroll
        for (int b = 0; b < NB; ++b)
          umma_bf16_x4_w(tmem + sr.stage * HEADS, umma_desc_sw128(base + ks.stage * P::kStage + b * kLtBox), 2,
                         umma_desc_sw128(base + P::kOffQ + b * HEADS * 128), 2, idesc_s, b);
        umma_commit_w(bar(kLtBarSFull + sr.stage));
        if (t == w.tiles - 1) umma_commit_w(bar(kLtBarQEmpty));
        ks.advance(P::kStages);
        sr.advance(2);
        return true;
      };
      ok = issue_s(0);
      for (int t = 0; t < w.tiles && ok; ++t) {
        if (t + 1 < w.tiles) ok = issue_s(t + 1);
        if (!ok) break;
        if (t == 0) {
          // the previous row's output must have been read out
          if (!mbar_wait_w(bar(kLtBarOEmpty), o_phase ^ 1)) { ok = false; break; }
          o_phase ^= 1;
        }
        if (!mbar_wait_w(bar(kLtBarPFull + pr.stage), pr.phase)) { ok = false; break; }
        tc_fence_after();
        const uint64_t p_desc = umma_desc_sw128(base + P::kOffP + pr.stage * P::kPBytes);
#pragma unroll
        for (int i = 0; i < NM; ++i)
          umma_bf16_x4_w(tmem + P::kTmemO + i * 2 * HEADS, lt_desc_mn(base + kr.stage * P::kStage + 2 * i * kLtBox), 128, p_desc, 2, idesc_o,
                         t > 0 ? 1u : 0u);
        umma_commit_w(bar(kLtBarKEmpty + kr.stage));
        umma_commit_w(bar(kLtBarPEmpty + pr.stage));
        if (t == w.tiles - 1) umma_commit_w(bar(kLtBarOFull));
        kr.advance(P::kStages);
        pr.advance(2);
      }
    }
    if (!ok && lane == 0) { misc[1] = 1; report_status(MDB_STATUS_WAIT_TIMEOUT); }
  } else {
    // ------------------------------------------------------------------- softmax
    const int tid = threadIdx.x, piece = tid & 7, my_head = tid >> 3;        // eight keys of a tile of head my_head (+ 16)
    const uint32_t lane_field = static_cast<uint32_t>(32 * warp) << 16;
    float* const turned = reinterpret_cast<float*>(mem + P::kOffS);
    float* const factor = reinterpret_cast<float*>(mem + P::kOffF);
    AtRing kr, sr, pr, prev;
    uint32_t o_phase = 0;
    while (walk.next(a, w)) {
      float m_ref[HG], l[HG];
#pragma unroll
      for (int g = 0; g < HG; ++g) { m_ref[g] = -INFINITY; l[g] = 0.f; }
      for (int t = 0; t < w.tiles; ++t) {
        wait(kLtBarSFull + sr.stage, sr.phase);
        __syncwarp();
        tc_fence_after();
        const int held = min(kLtKeys, w.keys - (w.tile0 + t) * kLtKeys);      // keys of the tile the token sees
        float* const mine = turned + sr.stage * HEADS * P::kSLd;
        {
          // row i of a product with M = 64 is on lane (i mod 16) + 32 (i div 16)
          const int key = 16 * warp + lane;
#pragma unroll
          for (int g = 0; g < HG; ++g) {
            float v[16];
            tmem_ld16(tmem + sr.stage * HEADS + 16 * g + lane_field, v);
            tmem_ld_wait();
            if (lane < 16) {
#pragma unroll
              for (int h = 0; h < 16; ++h) mine[(16 * g + h) * P::kSLd + key] = key < held ? v[h] * a.scale_log2 : -INFINITY;
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(kLtBarSEmpty + sr.stage));
        asm volatile("bar.sync 1, 128;" ::: "memory");
        float s[HG][8];
        int grow = 0;
#pragma unroll
        for (int g = 0; g < HG; ++g) {
          const float* row = mine + (16 * g + my_head) * P::kSLd + 8 * piece;
          *reinterpret_cast<float4*>(s[g]) = *reinterpret_cast<const float4*>(row);
          *reinterpret_cast<float4*>(s[g] + 4) = *reinterpret_cast<const float4*>(row + 4);
          float mx = s[g][0];
#pragma unroll
          for (int i = 1; i < 8; ++i) mx = fmaxf(mx, s[g][i]);
#pragma unroll
          for (int o = 1; o < 8; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
          float f = 1.f;
          if (mx > m_ref[g] + 8.f) {                      // (a tile holds at least one key; also the first time)
            f = ex2_approx(m_ref[g] - mx);
            m_ref[g] = mx;
            l[g] *= f;
            grow = 1;
          }
          if (piece == 0) factor[16 * g + my_head] = f;
        }
        int any;
        asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %1, 0;\n\tbarrier.cta.red.or.pred q, 1, 128, p;\n\tselp.s32 %0, 1, 0, q;\n\t}"
                     : "=r"(any) : "r"(grow) : "memory");
        if (any && t > 0) {
          // O is quiet once the last tile's products have completed
          wait(kLtBarPEmpty + prev.stage, prev.phase);
          __syncwarp();
          tc_fence_after();
#pragma unroll 1
          for (int c = 0; c < NM * 2 * HG; ++c) {
            float o[16];
            tmem_ld16(tmem + P::kTmemO + 16 * c + lane_field, o);
            tmem_ld_wait();
#pragma unroll
            for (int h = 0; h < 16; ++h) o[h] *= factor[16 * (c % HG) + h];
            tmem_stf16(tmem + P::kTmemO + 16 * c + lane_field, o);
          }
          tmem_st_wait();
        }
        wait(kLtBarPEmpty + pr.stage, pr.phase ^ 1);
        unsigned char* const p_tile = mem + P::kOffP + pr.stage * P::kPBytes;
#pragma unroll
        for (int g = 0; g < HG; ++g) {
          uint32_t hi[4], lo[4];
#pragma unroll
          for (int i = 0; i < 8; i += 2) {
            const float p0 = ex2_approx(s[g][i] - m_ref[g]), p1 = ex2_approx(s[g][i + 1] - m_ref[g]);
            l[g] += p0 + p1;
            const float h0 = bf16_round(p0), h1 = bf16_round(p1);
            hi[i / 2] = pack_bf16x2(h0, h1);
            lo[i / 2] = pack_bf16x2(p0 - h0, p1 - h1);
          }
          const int r = 16 * g + my_head, at = r * 128 + ((piece ^ (r & 7)) << 4);
          *reinterpret_cast<uint4*>(p_tile + at) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
          *reinterpret_cast<uint4*>(p_tile + HEADS * 128 + at) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        }
        if (held < kLtKeys) {
          // stale cache rows past the context must not reach O through 0 * (Inf or NaN)
          wait(kLtBarKFull + kr.stage, kr.phase);
          for (int i = tid; i < (kLtKeys - held) * NB * 8; i += 128) {
            const int c = i & 7, b = (i >> 3) % NB, r = held + (i >> 3) / NB;
            *reinterpret_cast<uint4*>(mem + kr.stage * P::kStage + b * kLtBox + r * 128 + c * 16) = make_uint4(0u, 0u, 0u, 0u);
          }
        }
        fence_async_smem();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(kLtBarPFull + pr.stage));
        prev = pr;
        kr.advance(P::kStages);
        sr.advance(2);
        pr.advance(2);
      }
      // ------------------------------------------------------------- output of the part
#pragma unroll
      for (int g = 0; g < HG; ++g) {
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) l[g] += __shfl_xor_sync(0xffffffffu, l[g], o);
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");      // the factors have been read
      const int64_t p0 = (static_cast<int64_t>(w.row) * a.nsplit + w.part) * a.heads + head0;
#pragma unroll
      for (int g = 0; g < HG; ++g) {
        const int h = 16 * g + my_head;
        if (piece == 0) {
          factor[h] = a.nsplit == 1 ? 1.0f / l[g] : 1.0f;
          if (a.nsplit > 1 && h < nh) a.part_ml[p0 + h] = make_float2(m_ref[g], l[g]);
        }
        // parts nobody computes
        if (a.nsplit > 1 && w.part == 0 && h < nh)
          for (int s = w.parts + piece; s < a.nsplit; s += 8)
            a.part_ml[(static_cast<int64_t>(w.row) * a.nsplit + s) * a.heads + head0 + h] = make_float2(-INFINITY, 0.f);
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");
      wait(kLtBarOFull, o_phase);
      __syncwarp();
      o_phase ^= 1;
      tc_fence_after();
#pragma unroll 1
      for (int i = 0; i < NM; ++i) {
        const int c = 128 * i + 32 * warp + lane;
#pragma unroll
        for (int g = 0; g < HG; ++g) {
          float hi[16], lo[16];
          tmem_ld16(tmem + P::kTmemO + i * 2 * HEADS + 16 * g + lane_field, hi);
          tmem_ld16(tmem + P::kTmemO + i * 2 * HEADS + HEADS + 16 * g + lane_field, lo);
          tmem_ld_wait();
#pragma unroll
          for (int h = 0; h < 16; ++h) {
            const int hh = 16 * g + h;
            if (hh < nh) {
              const float o = hi[h] + lo[h];
              if (a.nsplit == 1)
                static_cast<bf16*>(a.out)[(static_cast<int64_t>(w.row) * a.heads + head0 + hh) * WIDTH + c] = __float2bfloat16_rn(o * factor[hh]);
              else
                a.part_o[(p0 + hh) * WIDTH + c] = o;
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(kLtBarOEmpty));
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 5) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

template <int WIDTH, int HG>
static int latent_tc_run(const LatentArgs& a, cudaStream_t st) {
  using P = LtPlan<WIDTH, HG>;
  static PerDeviceOnce attr_once;
  const int dev = attr_once.slot();
  if (dev < 0) return MDB_ERR_CUDA;
  if (!attr_once.done[dev]) {
    if (cudaFuncSetAttribute(latent_attn_tc_kernel<WIDTH, HG>, cudaFuncAttributeMaxDynamicSharedMemorySize, P::kBytes) != cudaSuccess)
      return MDB_ERR_CUDA;
    attr_once.done[dev] = true;
  }
  CUtensorMap map_q, map_c;
  if (!get_tensor_map(a.q, static_cast<int64_t>(a.m) * a.heads, WIDTH, WIDTH, P::HEADS, &map_q)) return MDB_ERR_CUDA;
  if (!get_tensor_map(a.cache, static_cast<int64_t>(a.num_pages) * kPage, WIDTH, WIDTH, kLtKeys, &map_c)) return MDB_ERR_CUDA;
  const int groups = (a.heads + P::HEADS - 1) / P::HEADS, sms = at_sm_count();
  const int ctas = groups * (sms / groups > 0 ? sms / groups : 1);
  int rc = mdb_launch(latent_attn_tc_kernel<WIDTH, HG>, dim3(ctas), dim3(kLtThreads), P::kBytes, st, map_q, map_c, a);
  if (rc == MDB_OK && a.nsplit > 1) rc = mdb_launch(latent_combine_kernel, dim3(a.heads, a.m), dim3(128), 0, st, a);
  return rc;
}

// 32 heads per CTA where there are more than 16: a latent is then read once for all of them.
template <int WIDTH>
static int latent_tc_launch(const LatentArgs& a, cudaStream_t st) {
  return a.heads > 16 ? latent_tc_run<WIDTH, 2>(a, st) : latent_tc_run<WIDTH, 1>(a, st);
}

}  // namespace mdb
