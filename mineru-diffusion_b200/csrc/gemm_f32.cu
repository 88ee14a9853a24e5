// y = x W^T in true fp32, for the fp32 mode of the models that have one, on FMAs (a long k: gemm_f32_tc.cu).  Same
// three forms as the grouped tcgen05 kernel: plain, one weight per head (column blocks of x and y), one weight per expert (row
// tiles of 128).  GLU: half of a tile's weight rows are gate rows, the other half the up rows n further.
//
// 8 x 8 outputs per thread, operands as they lie in memory (k contiguous): no transposing, 16-byte cp.async into a ring and
// 16-byte reads out of it, 256 FMAs for 16 reads.  What bounds it: latency with two warps per scheduler, and the start and the end of
// a k this short (500 x 1536 x 384: 27 us, 22 TFLOP/s; at k 1024 33; a loop of 8 x 8 independent outputs reaches 114 FMA per cycle and
// SM scalar, 67 packed, which the register file bounds).  Rows of a stage are 36 floats long: the eight lanes that read eight
// neighbouring rows meet eight different groups of banks.
//
// An output is the sum of four chains over the blocks of 32 k, block by block in turn, whatever the tile: a row's bits do not depend on
// the other rows.  Where a CTA has four groups they take a chain each and add up in shared memory; one group runs the chains one
// behind the other.  So a tile of 64 x 64 has 256 threads, and 500 rows x 1024 columns already give 128 CTAs.
#include "mdb_common.cuh"

namespace mdb {

constexpr int kF32K = 32, kF32Ld = kF32K + 4;      // k of a group's stage; floats between rows
constexpr int kF32Chains = 4;                      // an output is the sum of four chains, whatever the tile

template <int BM, int BN, int TM, int TN, int KS, int STAGES>
struct F32Plan {
  static constexpr int TX = BN / TN, TY = BM / TM, kGroup = TX * TY, kThreads = kGroup * KS;
  static constexpr int kRows = BM + BN, kStage = KS * kRows * kF32Ld;                       // floats
  static constexpr int kSmemBytes = STAGES * kStage * 4;
  static_assert(KS == 1 || KS == kF32Chains, "a chain per group, or one behind another");
  static_assert(TX % 8 == 0 && (KS == 1 || TM % KS == 0), "eight lanes share a row of x; the last sums are dealt out by rows");
  static_assert(KS * BM * BN <= STAGES * kStage, "the groups' sums fit where the operands were");
};

template <int BM, int BN, int TM, int TN, int KS, int STAGES, bool GLU>
__global__ void __launch_bounds__(F32Plan<BM, BN, TM, TN, KS, STAGES>::kThreads, 1) gemm_f32_kernel(const mdb_gemm_args a) {
  using P = F32Plan<BM, BN, TM, TN, KS, STAGES>;
  extern __shared__ __align__(16) float f32_smem[];
  pdl_launch_dependents();
  pdl_wait();
  constexpr int kCols = GLU ? BN / 2 : BN;                 // output columns of a tile
  const int64_t row0 = static_cast<int64_t>(blockIdx.y) * BM;
  int64_t w_row0 = 0;
  int x_col = 0, y_col = 0;
  if (a.form == MDB_GEMM_HEADS) {
    w_row0 = static_cast<int64_t>(blockIdx.z) * a.n;
    x_col = blockIdx.z * a.k;
    y_col = blockIdx.z * a.n;
  } else if (a.form == MDB_GEMM_EXPERTS) {
    const int tile = static_cast<int>(row0 / kMoeTileRows);
    if (tile >= *a.num_tiles) return;
    w_row0 = static_cast<int64_t>(a.tile_expert[tile]) * a.n;
  }
  const float* x = static_cast<const float*>(a.x) + x_col;
  const float* w = static_cast<const float*>(a.w);
  const int n0 = blockIdx.x * kCols;
  const uint32_t smem = smem_u32(f32_smem);

  // 16-byte pieces of a stage: [group][x rows, then weight rows][eight of four k].  A thread fetches the same piece of the same NR
  // rows of every group and stage, so their addresses are worked out once; what lies outside arrives as zeros.
  constexpr int RS = P::kThreads / 8, NR = P::kRows / RS;
  static_assert(P::kRows % RS == 0, "whole rounds over the rows of a stage");
  const int piece = (threadIdx.x & 7) * 4;
  const float* src[NR];
  uint32_t live = 0;
#pragma unroll
  for (int q = 0; q < NR; ++q) {
    const int r = static_cast<int>(threadIdx.x >> 3) + RS * q;
    src[q] = static_cast<const float*>(a.w) + piece;
    if (r < BM) {
      if (row0 + r < a.m) {
        src[q] = x + (row0 + r) * a.ldx + piece;
        live |= 1u << q;
      }
    } else {
      const int rw = r - BM, up = GLU && rw >= kCols ? 1 : 0, col = n0 + rw - up * kCols;
      if (col < a.n) {
        src[q] = w + (w_row0 + col + (up ? a.n : 0)) * a.k + piece;
        live |= 1u << q;
      }
    }
  }
  const uint32_t dst0 = smem + ((threadIdx.x >> 3) * kF32Ld + piece) * 4;
  // KS 1: the blocks of 32 k in the order of the chains, chain c from step first_of(c) on
  const int blocks = (a.k + kF32K - 1) / kF32K;
  auto first_of = [&](int c) { return c * (blocks / kF32Chains) + min(c, blocks % kF32Chains); };
  auto block_of = [&](int step) {
    int c = 0;
#pragma unroll
    for (int i = 1; i < kF32Chains; ++i) c += step >= first_of(i) ? 1 : 0;
    return (step - first_of(c)) * kF32Chains + c;
  };
  auto fill = [&](int step) {
    const uint32_t dst = dst0 + (step % STAGES) * P::kStage * 4;
#pragma unroll
    for (int g = 0; g < KS; ++g) {
      const int k = (KS == 1 ? block_of(step) : step * KS + g) * kF32K;
#pragma unroll
      for (int q = 0; q < NR; ++q) {
        const bool in = (live >> q & 1u) && k + piece < a.k;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + (g * P::kRows + RS * q) * kF32Ld * 4),
                     "l"(in ? src[q] + k : static_cast<const float*>(a.w)), "r"(in ? 16u : 0u) : "memory");
      }
    }
  };

  const int group = threadIdx.x / P::kGroup, lid = threadIdx.x % P::kGroup, tx = lid % P::TX, ty = lid / P::TX;
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
  float sum[KS == 1 ? TM : 1][KS == 1 ? TN : 1];           // of the chains that have ended
  if (KS == 1) {
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) sum[KS == 1 ? i : 0][KS == 1 ? j : 0] = 0.f;
  }
  auto end_chain = [&]() {
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        sum[KS == 1 ? i : 0][KS == 1 ? j : 0] += acc[i][j];
        acc[i][j] = 0.f;
      }
  };
  const int steps = KS == 1 ? blocks : (a.k + KS * kF32K - 1) / (KS * kF32K);
  int chain = 1, chain_end = first_of(1);
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < steps) fill(s);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int s = 0; s < steps; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads();                                       // stage s is there for everyone, and stage s - 1 has been read
    if (s + STAGES - 1 < steps) fill(s + STAGES - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (KS == 1 && s == chain_end) {
      end_chain();
      chain_end = first_of(++chain);
    }
    const float* st = f32_smem + (s % STAGES) * P::kStage + group * P::kRows * kF32Ld;
    const float* xs = st + ty * kF32Ld;
    const float* ws = st + (BM + tx) * kF32Ld;
#pragma unroll 4
    for (int k = 0; k < kF32K; k += 4) {
      float4 xr[TM];
#pragma unroll
      for (int i = 0; i < TM; ++i) xr[i] = *reinterpret_cast<const float4*>(xs + i * P::TY * kF32Ld + k);
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const float4 wr = *reinterpret_cast<const float4*>(ws + j * P::TX * kF32Ld + k);
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(xr[i].x, wr.x, acc[i][j]);
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(xr[i].y, wr.y, acc[i][j]);
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(xr[i].z, wr.z, acc[i][j]);
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(xr[i].w, wr.w, acc[i][j]);
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  float* y = static_cast<float*>(a.y);
  auto leave = [&](int i, const float (&v)[TN]) {          // row i of the thread's outputs
    const int64_t row = row0 + i * P::TY + ty;
    if (row >= a.m) return;
#pragma unroll
    for (int j = 0; j < (GLU ? TN / 2 : TN); ++j) {
      const int col = n0 + j * P::TX + tx;
      if (col >= a.n) continue;
      float z = v[j];
      if (a.act == MDB_ACT_RELU2) { z = fmaxf(z, 0.f); z *= z; }
      if (a.act == MDB_ACT_SILU && col >= a.act_from) z /= 1.0f + expf(-z);
      if (GLU) z = fmaxf(z, 0.f) * v[GLU ? j + TN / 2 : 0];
      y[row * a.ldy + y_col + col] = z;
    }
  };
  if (KS == 1) {
    end_chain();
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      float v[TN];
#pragma unroll
      for (int j = 0; j < TN; ++j) v[j] = sum[KS == 1 ? i : 0][KS == 1 ? j : 0];
      leave(i, v);
    }
    return;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) f32_smem[((group * TM + i) * TN + j) * P::kGroup + lid] = acc[i][j];
  __syncthreads();
#pragma unroll
  for (int r = 0; r < (KS == 1 ? 1 : TM / KS); ++r) {
    const int i = group * (TM / KS) + r;
    float v[TN];
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      v[j] = 0.f;
#pragma unroll
      for (int g = 0; g < KS; ++g) v[j] += f32_smem[((g * TM + i) * TN + j) * P::kGroup + lid];
    }
    leave(i, v);
  }
}

template <int BM, int BN, int TM, int TN, int KS, int STAGES, bool GLU>
static int gemm_f32_run(const mdb_gemm_args& a, cudaStream_t st) {
  using P = F32Plan<BM, BN, TM, TN, KS, STAGES>;
  auto kernel = gemm_f32_kernel<BM, BN, TM, TN, KS, STAGES, GLU>;
  static PerDeviceOnce attr_once;
  const int dev = attr_once.slot();
  if (dev < 0) return MDB_ERR_CUDA;
  if (!attr_once.done[dev]) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, P::kSmemBytes) != cudaSuccess) return MDB_ERR_CUDA;
    attr_once.done[dev] = true;
  }
  const int cols = GLU ? BN / 2 : BN;
  const int64_t row_tiles = (static_cast<int64_t>(a.m) + BM - 1) / BM;
  const dim3 grid((a.n + cols - 1) / cols, static_cast<int>(row_tiles), a.form == MDB_GEMM_HEADS ? a.heads : 1);
  return mdb_launch(kernel, grid, dim3(P::kThreads), P::kSmemBytes, st, a);
}

// Rounds of a tile per SM times the FMA time of a tile per k: 128 cycles for 128 x 128 (a tenth less, it reads half as much through
// L2), 32 for 64 x 64, and 8 for 16 x 32, whose 4 x 4 outputs per thread are bound by shared memory at half the FMA rate.
template <bool GLU>
static int gemm_f32_dispatch(const mdb_gemm_args& a, cudaStream_t st) {
  const int64_t z = a.form == MDB_GEMM_HEADS ? a.heads : 1, n = GLU ? 2LL * a.n : a.n;
  const int64_t sms = at_sm_count();
  auto rounds = [&](int bm, int bn) {
    return (((static_cast<int64_t>(a.m) + bm - 1) / bm) * ((n + bn - 1) / bn) * z + sms - 1) / sms;
  };
  const int64_t wide = rounds(128, 128) * 115, mid = rounds(64, 64) * 32, narrow = rounds(16, 32) * 8;
  // grids reach 65535 row tiles: as many rows as tiles of 64 allowed
  if (narrow < mid && narrow < wide && a.m <= 16 * 65535) return gemm_f32_run<16, 32, 4, 4, 4, 4, GLU>(a, st);
  if (mid < wide) return gemm_f32_run<64, 64, 8, 8, 4, 3, GLU>(a, st);
  return gemm_f32_run<128, 128, 8, 8, 1, 4, GLU>(a, st);
}

static int gemm_f32_launch(const mdb_gemm_args& a, cudaStream_t st) {
  if (a.k % 16 != 0) return MDB_ERR_UNSUPPORTED;
  if ((static_cast<int64_t>(a.m) + 63) / 64 > 65535 || a.heads > 65535) return MDB_ERR_UNSUPPORTED;
  // From this k on on the tensor cores, by k alone, so that a row's bits do not depend on how many rows there are.  us on FMAs and there,
  // weights out of HBM, 1 / 8 / 16 / 500 rows:
  //   k 512,  n 64   4.1 4.7 / 4.3 4.9 / 4.4 4.7 / 6.5 5.4       n 1024  4.5 5.5 / 4.5 5.6 / 4.7 5.7 / 18 11
  //   k 640,  n 1024 5.6 6.4 / 5.5 6.5 / 5.7 6.5 / 22 12         n 4352  8.1 8.0 / 8.7 8.4 / 8.9 8.6 / 76 32
  //   k 768,  n 64   5.6 5.4 / 5.8 5.4 / 6.1 5.4 / 9.3 6.2       n 1024  6.2 6.4 / 6.5 6.6 / 6.8 6.6 / 25 14
  //   k 1024, n 1024 7.7 7.1 / 7.9 7.2 / 8.5 7.3 / 33 18         n 4352  12.0 10.2 / 12.7 10.6 / 13.1 10.8 / 117 45
  // What loses at 768 is a few rows of 1600 to 2048 columns whose weights are in L2 (6.0 6.3 / 6.6 6.7 / 6.6 6.7).
  if (a.k >= 768) return gemm_f32_tc_launch(a, st);
  return a.act == MDB_ACT_RELU_GLU ? gemm_f32_dispatch<true>(a, st) : gemm_f32_dispatch<false>(a, st);
}

}  // namespace mdb
