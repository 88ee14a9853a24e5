// Mixture of experts: group-limited top-k routing, the plan that lays the chosen (token, expert) pairs out by expert
// in tiles of 128 rows (the unit of the grouped GEMMs), and the row gather into that layout.
#include "mdb_common.cuh"

namespace mdb {

constexpr int kMoeTileRows = 128;      // rows of one expert start on a multiple of this
constexpr int kRouteWarps = 4;

// One warp per token.  Scores = softmax of the fp32 router logits over all experts; a group's score is its largest;
// the best `keep` groups stay in play; the `top` largest remaining scores win (ties to the lower index), and their
// weights are the scores divided by (their sum + 1e-20).
__global__ void __launch_bounds__(kRouteWarps * 32) moe_route_kernel(const mdb_moe_route_args a) {
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ float route_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t row = static_cast<int64_t>(blockIdx.x) * kRouteWarps + warp;
  if (row >= a.m) return;
  float* s = route_smem + warp * (a.experts + a.groups);
  float* gs = s + a.experts;
  if (a.row_slot != nullptr && a.row_slot[row] < 0) {       // padding row of a batch: routed nowhere
    for (int k = lane; k < a.top; k += 32) a.ids[row * a.top + k] = -1;
    return;
  }
  float mx = -INFINITY;
  for (int e = lane; e < a.experts; e += 32) {
    const float z = rows_at<float>(a.logits, row, e);
    s[e] = z;
    mx = fmaxf(mx, z);
  }
  mx = warp_max(mx);
  float sum = 0.f;
  for (int e = lane; e < a.experts; e += 32) {
    const float p = expf(s[e] - mx);
    s[e] = p;
    sum += p;
  }
  sum = warp_sum(sum);
  const float inv = 1.0f / sum;
  for (int e = lane; e < a.experts; e += 32) s[e] *= inv;
  __syncwarp();
  if (a.groups > 1 && a.keep < a.groups) {
    const int size = a.experts / a.groups;
    for (int g = lane; g < a.groups; g += 32) {
      float m = -INFINITY;
      for (int e = g * size; e < (g + 1) * size; ++e) m = fmaxf(m, s[e]);
      gs[g] = m;
    }
    __syncwarp();
    for (int g = lane; g < a.groups; g += 32) {
      int rank = 0;
      for (int o = 0; o < a.groups; ++o) rank += (gs[o] > gs[g] || (gs[o] == gs[g] && o < g)) ? 1 : 0;
      if (rank >= a.keep)
        for (int e = g * size; e < (g + 1) * size; ++e) s[e] = -1.0f;
    }
    __syncwarp();
  }
  float total = 0.f;
  for (int k = 0; k < a.top; ++k) {
    float bv = -2.0f;
    int bi = 0x7fffffff;
    for (int e = lane; e < a.experts; e += 32)
      if (s[e] > bv) { bv = s[e]; bi = e; }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
    }
    if (bi >= a.experts) { bi = 0; bv = 0.f; }          // only when every score is NaN
    total += bv;
    if (lane == 0) {
      a.ids[row * a.top + k] = bi;
      a.weights[row * a.top + k] = bv;
      s[bi] = -2.0f;
    }
    __syncwarp();
  }
  const float norm = 1.0f / (total + 1e-20f);
  for (int k = lane; k < a.top; k += 32) a.weights[row * a.top + k] *= norm;
}

// One CTA.  counts -> first row of every expert (multiples of 128) -> tile list -> a row for every (token, k) pair.
// The order of the rows of one expert is not fixed; every row's result is independent of its place.
// Bound by latencies one behind the other: the ids, the counts, the rows.  With up to KEEP ids per thread the count that a pair
// finds is its place among its expert's rows, and stays in a register with its expert: one walk over the ids and one over the rows'
// list; beyond that (KEEP 0) the ids are read twice.  With up to 64 experts (FEW) half a warp has one, lists its tiles and marks the rows
// that stay empty; with more of them a thread has one, and all rows are marked before they are given out.
// us, two walks and all rows marked, tiles listed by the scan / now:
//   8 experts, two a token:    1 token 2.2 / 1.8, 512 2.9 / 2.2, 1365 3.7 / 3.1, 4096 5.6 / 5.2
//   64 experts, six a token:   1 token 2.8 / 2.3, 128 3.5 / 3.4, 512 5.1 / 4.7, 2048 11.2 / 10.2, 4096 19.8 / 18.7
//   256 experts, eight a token: 1 token 4.4 / 3.0, 128 7.4 / 5.4, 512 9.5 / 8.3, 2048 17.9 / 16.7
constexpr int kPlanThreads = 1024, kPlanBatch = 8;
template <int KEEP, bool FEW>
__global__ void __launch_bounds__(kPlanThreads) moe_plan_kernel(const mdb_moe_plan_args a) {
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ int plan_smem[];
  int* count = plan_smem;              // [experts]
  int* first = plan_smem + a.experts;  // [experts]
  __shared__ int total_rows;
  const int n = a.m * a.top;
  int id[KEEP > 0 ? KEEP : 1], place[KEEP > 0 ? KEEP : 1];
  if (KEEP > 0) {
#pragma unroll
    for (int b = 0; b < KEEP; ++b) {
      const int i = static_cast<int>(threadIdx.x) + b * kPlanThreads;
      id[b] = a.ids[min(i, n - 1)];
      if (i >= n || id[b] < 0 || id[b] >= a.experts) id[b] = -1;
    }
  }
  for (int e = threadIdx.x; e < a.experts; e += kPlanThreads) count[e] = 0;
  __syncthreads();
  if (KEEP > 0) {
#pragma unroll
    for (int b = 0; b < KEEP; ++b) place[b] = id[b] >= 0 ? atomicAdd(&count[id[b]], 1) : 0;
  } else {
    for (int i0 = threadIdx.x; i0 < n; i0 += kPlanThreads * kPlanBatch) {
      int e[kPlanBatch];
#pragma unroll
      for (int b = 0; b < kPlanBatch; ++b) e[b] = i0 + b * kPlanThreads < n ? a.ids[i0 + b * kPlanThreads] : -1;
#pragma unroll
      for (int b = 0; b < kPlanBatch; ++b)
        if (e[b] >= 0 && e[b] < a.experts) atomicAdd(&count[e[b]], 1);
    }
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    // exclusive prefix of the tile counts, 32 experts at a time
    int base = 0;
    for (int e0 = 0; e0 < a.experts; e0 += 32) {
      const int e = e0 + threadIdx.x;
      const int tiles = e < a.experts ? (count[e] + kMoeTileRows - 1) / kMoeTileRows : 0;
      int incl = tiles;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (static_cast<int>(threadIdx.x) >= o) incl += v;
      }
      if (e < a.experts) first[e] = (base + incl - tiles) * kMoeTileRows;
      base += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (threadIdx.x == 0) {
      total_rows = base * kMoeTileRows;
      *a.num_tiles = base < a.max_tiles ? base : a.max_tiles;
    }
  }
  __syncthreads();
  const int cap = a.max_tiles * kMoeTileRows;
  // every expert's tiles, and the rows of its last one that stay empty
  constexpr int kLanes = FEW ? 16 : 1;
  for (int e = threadIdx.x / kLanes; e < a.experts; e += kPlanThreads / kLanes) {
    const int l = threadIdx.x % kLanes, r0 = first[e], r1 = r0 + count[e], r2 = r0 + (count[e] + kMoeTileRows - 1) / kMoeTileRows * kMoeTileRows;
    for (int t = r0 / kMoeTileRows + l; t < r2 / kMoeTileRows && t < a.max_tiles; t += kLanes) a.tile_expert[t] = e;
    if (FEW)
      for (int r = r1 + l; r < r2 && r < cap; r += kLanes) a.row_token[r] = -1;
  }
  if (!FEW) {
    for (int r = threadIdx.x; r < total_rows && r < cap; r += kPlanThreads) a.row_token[r] = -1;
    __syncthreads();
  }
  if (KEEP > 0) {
#pragma unroll
    for (int b = 0; b < KEEP; ++b) {
      const int i = static_cast<int>(threadIdx.x) + b * kPlanThreads;
      int slot = id[b] >= 0 ? first[id[b]] + place[b] : -1;
      if (slot >= cap) slot = -1;
      if (slot >= 0) a.row_token[slot] = i / a.top;
      if (i < n) a.slot[i] = slot;
    }
    return;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < a.experts; e += kPlanThreads) count[e] = 0;
  __syncthreads();
  for (int i0 = threadIdx.x; i0 < n; i0 += kPlanThreads * kPlanBatch) {
    int e[kPlanBatch];
#pragma unroll
    for (int b = 0; b < kPlanBatch; ++b) e[b] = i0 + b * kPlanThreads < n ? a.ids[i0 + b * kPlanThreads] : -1;
#pragma unroll
    for (int b = 0; b < kPlanBatch; ++b) {
      const int i = i0 + b * kPlanThreads;
      if (i >= n) break;
      int slot = -1;
      if (e[b] >= 0 && e[b] < a.experts) {
        slot = first[e[b]] + atomicAdd(&count[e[b]], 1);
        if (slot < cap) a.row_token[slot] = i / a.top;
        else slot = -1;
      }
      a.slot[i] = slot;
    }
  }
}

// Bound by memory and by a row's latencies, its place and its pieces; the next place is read meanwhile.  Few rows of up to 8 KB: a CTA per row, two
// pieces of 16 bytes in flight per thread.  Many: a warp per row, or per 4 KB of it, in eight rounds of 512 bytes that are all in flight, and in
// steps that shift a warp by 5/8 of a tile, as a tile's rows lie together and the rest of it is empty.
// us, a CTA per row and a piece in flight per thread / now (a warp per row in steps of whole tiles beside them):
//   rows of 4 KB:   2048 tokens of six of 64 experts 11.8 / 9.7 (9.7), 1000 6.2 / 5.8 (5.7), 300 of two of 8 2.0 / 2.1 (2.5)
//   rows of 8 KB:   700 of eight of 160 11.2 / 10.5 (13.4), 700 of two of 8 3.8 / 3.6 (5.1)
//   rows of 14 KB:  2048 of six of 64 48.5 / 38 (38), 300 of eight of 160 12.3 / 10.6 (14.7), 128 of two of 8 3.2 / 3.1 (4.9)
// (No __restrict__ on these pointers: a load the compiler may treat as invariant, like *num_tiles, moves above
// griddepcontrol.wait and then reads what the previous plan left.  Padding rows keep whatever they hold; nobody reads their results.)
__global__ void __launch_bounds__(128) moe_gather_few_kernel(const uint4* x, int64_t ldx, uint4* out, int chunks, const int32_t* row_token,
                                                             const int32_t* num_tiles) {
  pdl_launch_dependents();
  pdl_wait();
  const int rows = *num_tiles * kMoeTileRows;
  int r = blockIdx.x, t = r < rows ? row_token[r] : -1;
  while (r < rows) {
    uint4* dst = out + static_cast<int64_t>(r) * chunks;
    r += gridDim.x;
    const int next = r < rows ? row_token[r] : -1;
    if (t >= 0) {
      const uint4* src = x + static_cast<int64_t>(t) * ldx;
      for (int c = threadIdx.x; c < chunks; c += 256) {
        const uint4 v0 = src[c], v1 = src[min(c + 128, chunks - 1)];
        dst[c] = v0;
        if (c + 128 < chunks) dst[c + 128] = v1;
      }
    }
    t = next;
  }
}
__global__ void __launch_bounds__(128) moe_gather_kernel(const uint4* x, int64_t ldx, uint4* out, int chunks, int parts /* of a row */,
                                                         const int32_t* row_token, const int32_t* num_tiles) {
  pdl_launch_dependents();
  pdl_wait();
  const int rows = *num_tiles * kMoeTileRows, lane = threadIdx.x & 31, step = gridDim.x * 4, first = blockIdx.x * 4 + (threadIdx.x >> 5);
  int r = first / parts, part = first % parts;
  int t = r < rows ? row_token[r] : -1;
  while (r < rows) {
    const int c0 = part * 256 + lane;
    uint4* dst = out + static_cast<int64_t>(r) * chunks;
    r += step / parts;
    part += step % parts;
    if (part >= parts) {
      part -= parts;
      ++r;
    }
    const int next = r < rows ? row_token[r] : -1;
    if (t >= 0) {
      const uint4* src = x + static_cast<int64_t>(t) * ldx;
      uint4 v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = src[min(c0 + 32 * k, chunks - 1)];
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (c0 + 32 * k < chunks) dst[c0 + 32 * k] = v[k];
    }
    t = next;
  }
}

}  // namespace mdb

using namespace mdb;

extern "C" {

int mdb_moe_route(const mdb_moe_route_args* args, mdb_stream_t stream) {
  MDB_REQUIRE(args != nullptr, MDB_ERR_ARG);
  const mdb_moe_route_args a = *args;
  MDB_REQUIRE(a.m >= 0 && a.experts > 0 && a.top > 0 && a.groups > 0, MDB_ERR_ARG);
  if (a.m == 0) return MDB_OK;
  MDB_REQUIRE(a.experts % a.groups == 0 && a.keep > 0 && a.keep <= a.groups, MDB_ERR_ARG);
  MDB_REQUIRE(a.top <= a.keep * (a.experts / a.groups), MDB_ERR_ARG);
  MDB_REQUIRE(rows_present(a.logits) && a.ids && a.weights, MDB_ERR_ARG);
  const size_t smem = sizeof(float) * kRouteWarps * (a.experts + a.groups);
  MDB_REQUIRE(smem <= 48 * 1024, MDB_ERR_UNSUPPORTED);
  return mdb_launch(moe_route_kernel, dim3((a.m + kRouteWarps - 1) / kRouteWarps), dim3(kRouteWarps * 32), smem,
                    static_cast<cudaStream_t>(stream), a);
}

int mdb_moe_max_tiles(int m, int top, int experts) {
  if (m <= 0 || top <= 0 || experts <= 0) return 0;
  const int64_t pairs = static_cast<int64_t>(m) * top;
  const int64_t touched = pairs < experts ? pairs : experts;
  return static_cast<int>(touched + (pairs - touched) / kMoeTileRows);
}

int mdb_moe_plan(const mdb_moe_plan_args* args, mdb_stream_t stream) {
  MDB_REQUIRE(args != nullptr, MDB_ERR_ARG);
  const mdb_moe_plan_args a = *args;
  MDB_REQUIRE(a.m >= 0 && a.experts > 0 && a.top > 0 && a.max_tiles > 0, MDB_ERR_ARG);
  MDB_REQUIRE(a.ids && a.slot && a.row_token && a.tile_expert && a.num_tiles, MDB_ERR_ARG);
  MDB_REQUIRE(a.experts <= 4096 && static_cast<int64_t>(a.m) * a.top < (1 << 30), MDB_ERR_UNSUPPORTED);
  const int each = (a.m * a.top + kPlanThreads - 1) / kPlanThreads;
  // ids in registers as far as they pay: up to 12 a thread with few experts (5 of them: 6.0 us with two walks, 5.5; 12: 11.0, 10.2; 24: 18.7,
  // 18.2), up to four with many (8 of them: 10.7, 11.1).  An instance for more than there are costs 0.2 us an id.
  void (*const few)(mdb_moe_plan_args) = each < 1 || each > 12 ? moe_plan_kernel<0, true> : each <= 1 ? moe_plan_kernel<1, true>
                                         : each <= 4 ? moe_plan_kernel<4, true> : each <= 8 ? moe_plan_kernel<8, true> : moe_plan_kernel<12, true>;
  void (*const many)(mdb_moe_plan_args) = each < 1 || each > 4 ? moe_plan_kernel<0, false> : each <= 1 ? moe_plan_kernel<1, false> : moe_plan_kernel<4, false>;
  void (*const kernel)(mdb_moe_plan_args) = a.experts <= 64 ? few : many;
  return mdb_launch(kernel, dim3(1), dim3(kPlanThreads), sizeof(int) * 2 * a.experts, static_cast<cudaStream_t>(stream), a);
}

int mdb_moe_gather(int dtype, const void* x, int64_t ldx, void* out, int width, const int32_t* row_token,
                   const int32_t* num_tiles, int max_tiles, mdb_stream_t stream) {
  MDB_REQUIRE(width > 0 && max_tiles >= 0 && ldx >= width, MDB_ERR_ARG);
  if (max_tiles == 0) return MDB_OK;
  MDB_REQUIRE(x && out && row_token && num_tiles, MDB_ERR_ARG);
  MDB_REQUIRE(width % 8 == 0 && ldx % 8 == 0 && mdb_aligned16(x) && mdb_aligned16(out), MDB_ERR_ALIGN);
  const int per = 16 / (dtype == MDB_F32 ? 4 : 2), chunks = width / per, parts = (chunks + 255) / 256;      // elements of a piece, pieces
  const int64_t rows = static_cast<int64_t>(max_tiles) * kMoeTileRows;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const uint4* from = static_cast<const uint4*>(x);
  uint4* to = static_cast<uint4*>(out);
  int grid = 148 * 16;
  if (rows <= grid && chunks <= 512)      // (300 of two of 8, 14 KB: 4.7 us so, 4.0 by the other form)
    return mdb_launch(moe_gather_few_kernel, dim3(static_cast<unsigned>(rows)), dim3(128), 0, st, from, ldx / per, to, chunks, row_token, num_tiles);
  const int tile = kMoeTileRows / 4 * parts;      // CTAs that a tile's rows keep busy at once
  if (grid > tile) grid -= (grid - tile * 5 / 8) % tile;
  if ((rows * parts + 3) / 4 < grid) grid = static_cast<int>((rows * parts + 3) / 4);
  return mdb_launch(moe_gather_kernel, dim3(grid), dim3(128), 0, st, from, ldx / per, to, chunks, parts, row_token, num_tiles);
}

}  // extern "C"
