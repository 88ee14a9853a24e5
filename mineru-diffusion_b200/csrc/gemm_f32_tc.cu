// The fp32 products of gemm_f32.cu over a long k, on the 5th-generation tensor cores: plain, one weight per head, one weight per
// expert, and GLU (half of a tile's weight rows are gate rows, the other half the up rows n further).
//
// A number of 24 significant bits is the exact sum of three bf16 numbers (split3), so with a_i b_j exact in fp32
//   a b = a1 b1 + (a1 b2 + a2 b1) + (a1 b3 + a2 b2 + a3 b1) + (a2 b3 + a3 b2) + a3 b3,
// of which the last, below 2^-30 of a b, is left out: eight products on the tensor cores.  (The parts are cut off, not rounded, so
// those of size 2^-24 reach 2^-21 of a b, all of its sign.)  The sums by size go to accumulators of their own, and those of a1 b1,
// where the tensor cores' cutting off would show, end every 64 k and are added up in fp32 by threads.  The small ones are added to
// one another before they meet a large one: a row with a single number that is not zero has the error of one rounding.  Second parts come
// times 2^6, third parts times 2^12, so that small numbers keep all their bits; so a sum of size 2^-8 is 2^6 too large, the next two 2^12 and 2^18.
// Error of an output in 2^-24 of the sum of |a b|, largest and root mean square, beside chains of FMAs, k 768 / 1024 / 3072:
//   normal numbers   0.52, 0.085 (1.6, 0.24) / 0.48, 0.076 (1.8, 0.24) / 0.31, 0.052 (1.5, 0.24)
//   their sizes      4.0, 1.5 (7.7, 1.7) / 4.1, 1.6 (8.8, 2.1) / 4.4, 1.8 (13, 3.2): sums of one sign, cut off at every step
//   16 not zero      1.9, 0.30 (2.9, 0.37) / 1.9, 0.30 (2.4, 0.37) / 2.1, 0.31 (2.2, 0.38)
//   one not zero     0.99, 0.42 and the same for FMAs
// The first part of a number has its sign and is zero only where the number is (or below 2^-133); that of an infinity or NaN is the same, and
// its other parts are NaN.  So the sum of the a1 b1 is infinite or NaN where that of the a b is, and then the small sums are left
// out: such a result takes no longer than another.
//
// Tile: 128, 64 or 32 weight rows (the left operand) x 64 or 32 rows of x, k in chunks of 64.  Eight warps fetch rows of fp32 into
// registers a chunk ahead and leave their three parts in shared memory (K-major, 128-byte swizzle; the three parts of x one behind the
// other, so that one product takes a1 or a2 with b1 | b2 | b3, one a3 with b1 | b2), a warp issues the products, up to four warps add up.
// A chunk's small products go first: they wait for nothing, and meanwhile the chunk before's sums of a1 b1 are read.  Four chains
// over k, each a quarter of the chunks: a cluster of one, two or four CTAs shares them out, and they are added in the same order
// whoever ran them, so that the bits of a row do not depend on the other rows.
//
// What bounds it: bringing the operands in and turning them round.  A chunk of 128 x 64 outputs takes 2100 cycles, of which the
// products need 1030: its 48 KB come out of L2 (6 TB/s with all SMs), the parts are written to shared memory (72 KB) and read by the
// products (116 KB).  500 rows, n x k 4352 x 1024, 45 us with eight products and with six; with six 32 without the loads, 35 with a
// third of the parts' stores, 41 without splitting.  On FMAs it took 117; 1024 x 3072: 92 -> 35; 1024 x 1024: 33 -> 18.
// Few rows: a chunk's latency, so the weight rows of a tile are as few as still run all at once, and rows of x that are not there are
// not turned round (8 rows, 1024 x 1024, weights out of HBM: 9.4 us with 128 weight rows, 7.2 with 32; FMAs 7.9).  Registers, 128 a
// thread with 13 warps and 72 where two CTAs share an SM: 64 rows of x spill 16 bytes, tiles of 32 weight rows 40.  Not faster: two chunks
// ahead in registers (9.4 against 8.6 out of L2), weights asked into L2 in front of the dependency wait (8.7 against 7.5).
#include "mdb_common.cuh"

namespace mdb {

constexpr int kFtK = 64, kFtRows = 128, kFtChains = 4;
constexpr int kFtSumWarps = 4, kFtLoadWarps = 8, kFtMma = kFtSumWarps + kFtLoadWarps, kFtThreads = (kFtMma + 1) * 32;

template <int BN, int W>
struct FtPlan {
  static constexpr int kPartA = W * 128, kPartB = BN * 128, kStage = 3 * (kPartA + kPartB), kStages = 3;
  static constexpr int kSlot = W * BN * 4;                     // a chain's sums on their way to the other CTAs of the cluster
  static constexpr int kOffBars = kStages * kStage, kBytes = 1024 + kOffBars + 128;
  // tensor memory: a1 b1 of a chunk | of size 2^-8 | of size 2^-16 | of size 2^-24 of a chain | sums of the chains before
  static constexpr uint32_t kSum = 4 * BN, kTmemCols = BN == 32 ? 256 : 512;
  static_assert(2 * kSlot <= kStages * kStage && kBytes <= 227 * 1024 && 5 * BN <= kTmemCols, "memory of the fp32 product");
  // a product always takes 128 weight rows: behind the W of a part it finds others, whose sums nobody reads
  static_assert(2 * kPartA + kFtRows * 128 <= kStage, "a product's reads end in its stage");
};
enum { kFtFull = 0, kFtEmpty = 3, kFtDFull = 6, kFtDEmpty = 7, kFtBars = 8 };

__device__ __align__(32) const float kFtZeros[8] = {};
// Eight floats, in one load where they lie on a boundary of 32 bytes (two of 16 bytes read every 32-byte sector twice)
__device__ __forceinline__ void ldg_f8(const float* p, bool wide, f32x2 (&v)[4]) {
  asm volatile(
      "{\n\t.reg .pred t;\n\tsetp.ne.b32 t, %5, 0;\n\t"
      "@t ld.global.v4.b64 {%0, %1, %2, %3}, [%4];\n\t"
      "@!t ld.global.v2.b64 {%0, %1}, [%4];\n\t@!t ld.global.v2.b64 {%2, %3}, [%4 + 16];\n\t}"
      : "=&l"(v[0]), "=&l"(v[1]), "=&l"(v[2]), "=&l"(v[3]) : "l"(p), "r"(static_cast<uint32_t>(wide)) : "memory");
}
template <bool GLU>
__device__ __forceinline__ float f32_activated(const mdb_gemm_args& a, float z, float up, int col) {
  if (a.act == MDB_ACT_RELU2) { z = fmaxf(z, 0.f); z *= z; }
  if (a.act == MDB_ACT_SILU && col >= a.act_from) z /= 1.0f + expf(-z);
  return GLU ? fmaxf(z, 0.f) * up : z;
}
template <int BN, int W, bool GLU>
__global__ void __launch_bounds__(kFtThreads, W == 32 ? 2 : 1) gemm_f32_tc_kernel(const mdb_gemm_args a, const int ctas /* of a cluster */) {
  using P = FtPlan<BN, W>;
  extern __shared__ __align__(1024) unsigned char ft_smem_raw[];
  const uint32_t raw = smem_u32(ft_smem_raw), base = (raw + 1023u) & ~1023u;
  unsigned char* mem = ft_smem_raw + (base - raw);
  const uint32_t bars = base + P::kOffBars;
  volatile uint32_t* misc = reinterpret_cast<volatile uint32_t*>(mem + P::kOffBars + 8 * kFtBars);      // tensor memory base, abort flag
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = ctas > 1 ? static_cast<int>(cluster_ctarank()) : 0;
  constexpr int kCols = GLU ? W / 2 : W, kSumWarps = W / 32;       // output columns of a tile; warps that add up
  const int n0 = static_cast<int>(blockIdx.x) / ctas * kCols;
  const int64_t row0 = static_cast<int64_t>(blockIdx.y) * BN;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kFtBars; ++s) mbar_init(bars + 8 * s, s < kFtEmpty ? kFtLoadWarps : (s < kFtDEmpty ? 1 : kSumWarps));
    misc[1] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kFtMma) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(const_cast<uint32_t*>(&misc[0]))), "r"(P::kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  pdl_wait();
  int64_t w_row0 = 0;
  int x_col = 0, y_col = 0;
  bool live = true;
  if (a.form == MDB_GEMM_HEADS) {
    w_row0 = static_cast<int64_t>(blockIdx.z) * a.n;
    x_col = blockIdx.z * a.k;
    y_col = blockIdx.z * a.n;
  } else if (a.form == MDB_GEMM_EXPERTS) {
    const int tile = static_cast<int>(row0 / kMoeTileRows);
    live = tile < *a.num_tiles;
    if (live) w_row0 = static_cast<int64_t>(a.tile_expert[tile]) * a.n;
  }
  const float* const x = static_cast<const float*>(a.x) + x_col;
  const float* const w = static_cast<const float*>(a.w) + w_row0 * a.k;
  // barriers and tensor memory are there; the load warps come here with their first chunk under way
  auto ready = [&]() {
    tc_fence_before();
    asm volatile("bar.sync 2, %0;" ::"n"(kFtThreads) : "memory");
    tc_fence_after();
    pdl_launch_dependents();
    return misc[0];
  };
  // A wait that runs out raises the abort flag; the roles then walk to the end without waiting for long again.
  auto wait = [&](int s, uint32_t parity) {
    uint32_t done;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(done) : "r"(bars + 8 * s), "r"(parity) : "memory");
    if (done || misc[1] != 0) return;
    if (!mbar_wait(bars + 8 * s, parity)) {
      misc[1] = 1;
      report_status(MDB_STATUS_WAIT_TIMEOUT);
    }
  };
  // chain c: chunks [first_of(c), first_of(c + 1)); this CTA's chains are one behind the other
  const int chunks = (a.k + kFtK - 1) / kFtK;
  auto first_of = [&](int c) { return (c * chunks + kFtChains - 1) / kFtChains; };
  const int chain0 = rank * (kFtChains / ctas), chain1 = chain0 + kFtChains / ctas;
  const int begin = live ? first_of(chain0) : 0, end = live ? first_of(chain1) : 0;
  // what a CTA leaves for the cluster: the first one the sum of its chains, the others each chain by itself
  auto slots_of = [&](int r) {
    int n = 0;
    for (int c = r * (kFtChains / ctas); c < (r + 1) * (kFtChains / ctas); ++c) n += first_of(c + 1) > first_of(c) ? 1 : 0;
    return r == 0 ? min(n, 1) : n;
  };

  if (warp == kFtMma) {
    // ---------------------------------------------------------------- products
    const uint32_t tmem = ready();
    const uint32_t id1 = umma_idesc_bf16(BN), id2 = umma_idesc_bf16(2 * BN), id3 = umma_idesc_bf16(3 * BN);
    uint32_t phase = 0, used = 0;      // a bit per stage; chunks so far
    int stage = 0;
    for (int c = chain0; c < chain1; ++c) {
      const int c0 = first_of(c), c1 = live ? first_of(c + 1) : c0;
      for (int i = c0; i < c1; ++i) {
        if (i == c0) wait(kFtDEmpty, (used & 1u) ^ 1u);      // the small sums of the chain before have been read
        wait(kFtFull + stage, phase >> stage & 1u);
        __syncwarp();
        tc_fence_after();
        if (misc[1] != 0) break;
        const uint32_t at = base + stage * P::kStage;
        const uint64_t b1 = umma_desc_sw128(at + 3 * P::kPartA);
        const uint64_t a1 = umma_desc_sw128(at), a2 = umma_desc_sw128(at + P::kPartA), a3 = umma_desc_sw128(at + 2 * P::kPartA);
#pragma unroll
        for (int s = 0; s < kFtK / 16; ++s) {
          umma_bf16_w(tmem + BN, a2 + 2 * s, b1 + 2 * s, id3, i == c0 && s == 0 ? 0u : 1u);
          umma_bf16_w(tmem + 2 * BN, a3 + 2 * s, b1 + 2 * s, id2, 1u);
        }
        if (i > c0) {      // the chunk before's sums of a1 b1 have been read
          wait(kFtDEmpty, (used & 1u) ^ 1u);
          __syncwarp();
          tc_fence_after();
        }
        umma_bf16_w(tmem, a1, b1, id1, 0u);
        umma_bf16_w(tmem + BN, a1, b1 + (P::kPartB >> 4), id2, 1u);
#pragma unroll
        for (int s = 1; s < kFtK / 16; ++s) umma_bf16_w(tmem, a1 + 2 * s, b1 + 2 * s, id3, 1u);
        umma_commit_w(bars + 8 * (kFtEmpty + stage));
        umma_commit_w(bars + 8 * kFtDFull);
        phase ^= 1u << stage;
        ++used;
        stage = stage + 1 == P::kStages ? 0 : stage + 1;
      }
    }
  } else if (warp >= kFtSumWarps) {
    // ------------------------------------------------------------------ operands
    // 32 bytes of k of a row per lane, eight lanes a row; a thread has the same piece of NR rows of every chunk
    constexpr int NR = (W + BN) / 32;
    const int tid = threadIdx.x - kFtSumWarps * 32, piece = tid & 7, r0 = tid >> 3;
    const float* const x0 = x + (row0 + r0) * a.ldx + 8 * piece;
    const float* const w0 = w + static_cast<int64_t>(n0 + r0 + (GLU && kCols < 32 && r0 >= kCols ? a.n - kCols : 0)) * a.k + 8 * piece;
    uint32_t there = 0;
#pragma unroll
    for (int q = 0; q < NR; ++q) {
      const int r = r0 + 32 * q;
      if (r < W ? n0 + r % kCols < a.n : row0 + r - W < a.m) there |= 1u << q;
    }
    const float* const zeros = kFtZeros;      // what lies outside
    const bool wide = ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 31) == 0;      // rows of 16 k, or 8 of x
    f32x2 v[NR][4];
    auto fetch = [&](int q, int chunk) {
      const int k = chunk * kFtK;
      const float* from = 32 * q >= W ? x0 + (32 * q - W) * a.ldx
                                             : w0 + (static_cast<int64_t>(GLU && kCols >= 32 && 32 * q >= kCols ? a.n - kCols : 0) + 32 * q) * a.k;
      ldg_f8((there >> q & 1u) && chunk < end && k + 8 * piece < a.k ? from + k : zeros, wide, v[q]);
    };
#pragma unroll
    for (int q = 0; q < NR; ++q) fetch(q, begin);
    ready();
    int stage = 0;
    uint32_t phase = 0;
    const uint32_t dst0 = base + r0 * 128 + ((piece ^ (r0 & 7)) << 4);
    for (int i = begin; i < end; ++i) {
      wait(kFtEmpty + stage, (phase >> stage & 1u) ^ 1u);
      const uint32_t dst = dst0 + stage * P::kStage;
#pragma unroll
      for (int q = 0; q < NR; ++q) {
        if (32 * q >= W && !(there >> q & 1u)) continue;      // a row of x that is not there: its sums go nowhere
        uint32_t p[4][3];
#pragma unroll
        for (int e = 0; e < 4; ++e) split3(v[q][e], p[e]);
        fetch(q, i + 1);
        const bool is_w = 32 * q < W;
        const uint32_t to = dst + (is_w ? 32 * q * 128 : 3 * P::kPartA + (32 * q - W) * 128);
#pragma unroll
        for (int e = 0; e < 3; ++e)
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(to + e * (is_w ? P::kPartA : P::kPartB)), "r"(p[0][e]), "r"(p[1][e]),
                       "r"(p[2][e]), "r"(p[3][e]) : "memory");
      }
      fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(bars + 8 * (kFtFull + stage));
      phase ^= 1u << stage;
      stage = stage + 1 == P::kStages ? 0 : stage + 1;
    }
  } else if (warp >= kSumWarps) {
    ready();
  } else {
    // ---------------------------------------------------------------------- sums
    const uint32_t lanes = ready() + (static_cast<uint32_t>(32 * warp) << 16);
    float acc[BN];
    uint32_t used = 0;
    bool parked = false;
    auto add = [&](uint32_t col) {
#pragma unroll
      for (int j = 0; j < BN; j += 32) {
        float d[2][16];
        tmem_ld16(lanes + col + j, d[0]);
        tmem_ld16(lanes + col + j + 16, d[1]);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 32; ++e) acc[j + e] += d[e / 16][e % 16];
      }
    };
    // a chain's small sums, smallest first, each kSplitUp times too large against the one before; beside a sum that is not finite they
    // say nothing
    auto add_small = [&]() {
      constexpr float kDown = 1.0f / kSplitUp;
#pragma unroll
      for (int j = 0; j < BN; j += 16) {
        float t[16], u[16];
        tmem_ld16(lanes + 3 * BN + j, t);
        tmem_ld16(lanes + 2 * BN + j, u);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 16; ++e) t[e] = fmaf(t[e], kDown, u[e]);
        tmem_ld16(lanes + BN + j, u);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 16; ++e)
          if (isfinite(acc[j + e])) acc[j + e] = fmaf(fmaf(t[e], kDown, u[e]), kDown, acc[j + e]);
      }
    };
    for (int c = chain0; c < chain1; ++c) {
      const int c0 = first_of(c), c1 = live ? first_of(c + 1) : c0;
      if (c1 <= c0) continue;
#pragma unroll
      for (int j = 0; j < BN; ++j) acc[j] = 0.f;
      for (int i = c0; i < c1; ++i) {
        wait(kFtDFull, used & 1u);
        __syncwarp();
        tc_fence_after();
        add(0);
        if (i == c1 - 1) {
          add_small();
          if (rank == 0 && parked) add(P::kSum);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bars + 8 * kFtDEmpty);
        ++used;
      }
      const bool last = c == chain1 - 1 || first_of(chain1) == c1;
      if (!last) {      // the operands' memory is still in use: these sums wait in tensor memory
#pragma unroll
        for (int j = 0; j < BN; j += 16) tmem_stf16(lanes + P::kSum + j, acc + j);
        tmem_st_wait();
        parked = true;
      }
    }
    // every product of this CTA is done: its operands' memory takes the sums
    if (ctas > 1 && end > begin) {
#pragma unroll 1
      for (int slot = rank > 0 && parked ? 1 : 0; slot >= 0; --slot) {
        float* to = reinterpret_cast<float*>(mem + slot * P::kSlot) + 32 * warp + lane;
#pragma unroll
        for (int j = 0; j < BN; ++j) {
          to[j * W] = acc[j];
          acc[j] = 0.f;
        }
        if (slot > 0) add(P::kSum);
      }
    }
    if (ctas == 1 && live) {
      // a column per thread: 32 neighbours of a row at once
      const int col = (32 * warp + lane) % kCols, out = n0 + col;
      float* up = reinterpret_cast<float*>(mem) + col;
      if (GLU) {
        if (32 * warp + lane >= kCols) {
#pragma unroll
          for (int j = 0; j < BN; ++j) up[j * kCols] = acc[j];
        }
        asm volatile("bar.sync 1, %0;" ::"n"(kSumWarps * 32) : "memory");
      }
      if (out < a.n && (!GLU || 32 * warp + lane < kCols) && misc[1] == 0) {
        float* const y = static_cast<float*>(a.y) + row0 * a.ldy + y_col + out;
        const int rows = static_cast<int>(min(static_cast<int64_t>(BN), a.m - row0));
#pragma unroll
        for (int j = 0; j < BN; ++j)
          if (GLU) acc[j] = fmaxf(acc[j], 0.f) * up[j * kCols];
        if (a.act == MDB_ACT_RELU2) {
#pragma unroll
          for (int j = 0; j < BN; ++j) {
            acc[j] = fmaxf(acc[j], 0.f);
            acc[j] *= acc[j];
          }
        } else if (a.act == MDB_ACT_SILU && out >= a.act_from) {
#pragma unroll
          for (int j = 0; j < BN; ++j) acc[j] = f32_activated<GLU>(a, acc[j], 0.f, out);
        }
        float* at = y;
        if (rows == BN) {
#pragma unroll
          for (int j = 0; j < BN; ++j, at += a.ldy) *at = acc[j];
        } else {
#pragma unroll
          for (int j = 0; j < BN; ++j, at += a.ldy)
            if (j < rows) *at = acc[j];
        }
      }
    }
  }
  tc_fence_before();
  if (ctas > 1) cluster_sync_all();
  else __syncthreads();
  tc_fence_after();
  if (warp == kFtMma) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(misc[0]), "r"(P::kTmemCols));
  if (ctas > 1 && live && misc[1] == 0) {
    // this CTA's rows of the tile: the sums that every CTA has left, in their order
    uint32_t from[kFtChains];
    int slots = 0;
    for (int r = 0; r < ctas; ++r) {
      const int n = slots_of(r);
      for (int s = 0; s < n; ++s) {
#pragma unroll
        for (int i = 0; i < kFtChains; ++i)
          if (i == slots) from[i] = map_to_cta(base + s * P::kSlot, static_cast<uint32_t>(r));
        ++slots;
      }
    }
    constexpr int kGroups = kFtThreads / kCols;                     // rows at a time
    const int col = threadIdx.x % kCols, g = threadIdx.x / kCols, out = n0 + col;
    float* y = static_cast<float*>(a.y) + row0 * a.ldy + y_col + out;
    const int rows = static_cast<int>(min(static_cast<int64_t>(BN / ctas * (rank + 1)), a.m - row0));
    if (g < kGroups && out < a.n) {
#pragma unroll 2
      for (int j = BN / ctas * rank + g; j < rows; j += kGroups) {
        float z[kFtChains][GLU ? 2 : 1];
#pragma unroll
        for (int i = 0; i < kFtChains; ++i)
#pragma unroll
          for (int h = 0; h < (GLU ? 2 : 1); ++h) {
            z[i][h] = 0.f;
            if (i < slots)
              asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(z[i][h]) : "r"(from[i] + (j * W + h * kCols + col) * 4) : "memory");
          }
        float t[2] = {z[0][0], z[0][GLU ? 1 : 0]};
#pragma unroll
        for (int i = 1; i < kFtChains; ++i)
          if (i < slots) {
            t[0] += z[i][0];
            t[1] += z[i][GLU ? 1 : 0];
          }
        y[j * a.ldy] = f32_activated<GLU>(a, t[0], t[1], out);
      }
    }
  }
  // no CTA leaves while another may still read its shared memory; nothing is handed over here, and what a thread has read it has used
  if (ctas > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}

template <int BN, int W, bool GLU>
static int gemm_f32_tc_run(const mdb_gemm_args& a, int ctas, cudaStream_t st) {
  using P = FtPlan<BN, W>;
  auto kernel = gemm_f32_tc_kernel<BN, W, GLU>;
  static PerDeviceOnce attr_once;
  const int dev = attr_once.slot();
  if (dev < 0) return MDB_ERR_CUDA;
  if (!attr_once.done[dev]) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, P::kBytes) != cudaSuccess) return MDB_ERR_CUDA;
    attr_once.done[dev] = true;
  }
  const int cols = GLU ? W / 2 : W;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((a.n + cols - 1) / cols * ctas, static_cast<unsigned>((static_cast<int64_t>(a.m) + BN - 1) / BN), a.form == MDB_GEMM_HEADS ? a.heads : 1);
  cfg.blockDim = dim3(kFtThreads);
  cfg.dynamicSmemBytes = P::kBytes;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = ctas;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = g_opt_pdl ? attr : attr + 1;
  cfg.numAttrs = (g_opt_pdl ? 1 : 0) + (ctas > 1 ? 1 : 0);
  return cudaLaunchKernelEx(&cfg, kernel, a, ctas) == cudaSuccess ? MDB_OK : MDB_ERR_CUDA;
}

// Rounds of the CTAs times the time of one, in hundredths of a us as measured: a chunk, and what is beside it in clusters of one,
// two and four (of a cluster of two the second CTA leaves two chains).  Clusters of four do not fill every SM: 33 run at once on 148.
// Of 540 sizes (1 to 1000 rows, 64 to 8192 columns, k 768 to 3072) the form taken was within 8 % of the best of the twelve.
struct FtForm { int rows, weights, chunk, rest[3]; };
constexpr FtForm kFtForms[4] = {
    {64, 128, 108, {530, 900, 790}}, {32, 128, 87, {390, 610, 530}}, {32, 64, 70, {390, 510, 510}}, {32, 32, 58, {440, 540, 520}}};
template <bool GLU>
static int gemm_f32_tc_dispatch(const mdb_gemm_args& a, cudaStream_t st) {
  const int chunks = (a.k + kFtK - 1) / kFtK;
  const int64_t n = GLU ? 2LL * a.n : a.n, sms = at_sm_count();
  int64_t best = INT64_MAX;
  int form = 0, ctas = 1;
  for (int f = 0; f < 4; ++f) {
    const FtForm& p = kFtForms[f];
    if (a.m > p.rows * 65535LL) continue;
    const int64_t tiles = (n + p.weights - 1) / p.weights * (a.form == MDB_GEMM_HEADS ? a.heads : 1) * ((static_cast<int64_t>(a.m) + p.rows - 1) / p.rows);
    for (int lg = 0; lg < 3; ++lg) {
      const int c = 1 << lg;
      const int64_t at_once = max(lg == 2 ? sms / 4 - 4 : sms / c, static_cast<int64_t>(1));
      const int64_t time = (tiles + at_once - 1) / at_once * ((chunks + c - 1) / c * p.chunk + p.rest[lg]);
      if (time < best) { best = time; form = f; ctas = c; }
    }
  }
  switch (form) {
    case 0: return gemm_f32_tc_run<64, 128, GLU>(a, ctas, st);
    case 1: return gemm_f32_tc_run<32, 128, GLU>(a, ctas, st);
    case 2: return gemm_f32_tc_run<32, 64, GLU>(a, ctas, st);
    default: return gemm_f32_tc_run<32, 32, GLU>(a, ctas, st);
  }
}

static int gemm_f32_tc_launch(const mdb_gemm_args& a, cudaStream_t st) {
  return a.act == MDB_ACT_RELU_GLU ? gemm_f32_tc_dispatch<true>(a, st) : gemm_f32_tc_dispatch<false>(a, st);
}

}  // namespace mdb
