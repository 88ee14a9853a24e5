// Causal attention over cached latents: every query head of a token reads the same latent row of a key, which stands
// for its key and its value alike (the per-head key projection is folded into the query, the per-head value
// projection follows the attention), so a key costs one latent row of memory traffic for all heads.
//
//   latent_attn_tc_kernel    bf16, widths of 128 to 512 (latent_attention_tc.cu); parts of a context are merged by
//                            latent_combine_kernel.
//   latent_attn_rows_kernel  fp32, and widths the first kernel does not take: one CTA per (token, head), a warp per key.
#include "mdb_common.cuh"

namespace mdb {

struct LatentArgs {
  const void* q;              // [m][heads][width]
  const void* cache;          // [pages * 256][width]
  void* out;                  // [m][heads][width]
  float* part_o;              // [m][nsplit][heads][width]
  float2* part_ml;            // [m][nsplit][heads]   (max in log2 units, sum)
  const int32_t* table;
  const int32_t* row_seq;
  const int32_t* row_pos;     // position of the row's token; -1: padding row
  int table_stride, num_pages, m, heads, width, nsplit;
  float scale_log2;
};

__device__ __forceinline__ int64_t latent_slot(const LatentArgs& a, const int32_t* table, int pos) {
  int page = pos / kPage < a.table_stride ? table[pos / kPage] : -1;
  if (page < 0 || page >= a.num_pages) {
    report_status(MDB_STATUS_BAD_PAGE);
    page = 0;
  }
  return static_cast<int64_t>(page) * kPage + pos % kPage;
}

__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm4_t(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// One CTA per (head, row): the key-range parts of a context weighted by their maxima.  Every warp works out the weights (a part
// per lane and round), then four parts are in flight at a time: part by part, a maximum and the row behind it are two latencies.
__global__ void __launch_bounds__(128) latent_combine_kernel(const LatentArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  const int row = blockIdx.y, head = blockIdx.x, lane = threadIdx.x & 31;
  if (a.row_pos[row] < 0) return;
  const int64_t p0 = static_cast<int64_t>(row) * a.nsplit * a.heads + head;
  float mx = -INFINITY, l = 0.f;
  for (int s = lane; s < a.nsplit; s += 32) mx = fmaxf(mx, a.part_ml[p0 + static_cast<int64_t>(s) * a.heads].x);
  mx = warp_max(mx);
  for (int s = lane; s < a.nsplit; s += 32) {
    const float2 ml = a.part_ml[p0 + static_cast<int64_t>(s) * a.heads];
    l += ml.y * exp2f(ml.x - mx);
  }
  const float inv = 1.0f / warp_sum(l);
  bf16* out = static_cast<bf16*>(a.out) + (static_cast<int64_t>(row) * a.heads + head) * a.width;
  for (int c = threadIdx.x * 4; c < a.width; c += 512) {
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int s0 = 0; s0 < a.nsplit; s0 += 4) {
      float w[4];
      float4 v[4];
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        const float m = s0 + s < a.nsplit ? a.part_ml[p0 + static_cast<int64_t>(s0 + s) * a.heads].x : -INFINITY;
        w[s] = m == -INFINITY ? 0.f : exp2f(m - mx) * inv;
        v[s] = make_float4(0.f, 0.f, 0.f, 0.f);            // an empty part left its accumulator unwritten
        if (m != -INFINITY) v[s] = *reinterpret_cast<const float4*>(a.part_o + (p0 + static_cast<int64_t>(s0 + s) * a.heads) * a.width + c);
      }
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        o.x = fmaf(w[s], v[s].x, o.x); o.y = fmaf(w[s], v[s].y, o.y); o.z = fmaf(w[s], v[s].z, o.z); o.w = fmaf(w[s], v[s].w, o.w);
      }
    }
    act_store4(out + c, o);
  }
}

// One CTA of four warps per (head, row); warp w takes keys w, w + 4, ...; a lane owns every 32nd float4 group of four
// channels.  NV = channels per lane / 4.  What bounds it: every head reads the latents for itself, out of L2 (500 rows of 8 heads, width
// 256: 1 GB, 116 us; 132 with one key at a time, whose row, sum over lanes and weight follow one another).
template <typename T, int NV>
__global__ void __launch_bounds__(128) latent_attn_rows_kernel(const LatentArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float sm[4], sl[4];
  extern __shared__ float rows_o[];        // [4][width]
  const int row = blockIdx.y, head = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int pos = a.row_pos[row];
  if (pos < 0) return;
  const int32_t* table = a.table + static_cast<int64_t>(a.row_seq[row]) * a.table_stride;
  const T* q = static_cast<const T*>(a.q) + (static_cast<int64_t>(row) * a.heads + head) * a.width;
  float4 qv[NV], o[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    qv[i] = o[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    const int c = (lane + 32 * i) * 4;
    if (c < a.width) qv[i] = act_load4(q + c);
  }
  float m = -INFINITY, l = 0.f;
  // several keys at a time, as registers allow: their rows are in flight together and share a new maximum
  constexpr int KEYS = NV <= 2 ? 4 : NV <= 4 ? 2 : 1;
  for (int key = warp; key <= pos; key += 4 * KEYS) {
    float4 kv[KEYS][NV];
#pragma unroll
    for (int j = 0; j < KEYS; ++j) {
      const T* kr = static_cast<const T*>(a.cache) + latent_slot(a, table, min(key + 4 * j, pos)) * a.width;
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        kv[j][i] = make_float4(0.f, 0.f, 0.f, 0.f);
        const int c = (lane + 32 * i) * 4;
        if (c < a.width) kv[j][i] = act_load4(kr + c);
      }
    }
    float s[KEYS], m_new = m;
#pragma unroll
    for (int j = 0; j < KEYS; ++j) {
      s[j] = 0.f;
#pragma unroll
      for (int i = 0; i < NV; ++i) s[j] += qv[i].x * kv[j][i].x + qv[i].y * kv[j][i].y + qv[i].z * kv[j][i].z + qv[i].w * kv[j][i].w;
    }
#pragma unroll
    for (int j = 0; j < KEYS; ++j) {
      s[j] = key + 4 * j <= pos ? warp_sum(s[j]) * a.scale_log2 : -INFINITY;
      m_new = fmaxf(m_new, s[j]);
    }
    const float f = exp2f(m - m_new);
    m = m_new;
    l *= f;
#pragma unroll
    for (int i = 0; i < NV; ++i) { o[i].x *= f; o[i].y *= f; o[i].z *= f; o[i].w *= f; }
#pragma unroll
    for (int j = 0; j < KEYS; ++j) {
      const float p = exp2f(s[j] - m);
      l += p;
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        o[i].x = fmaf(p, kv[j][i].x, o[i].x); o[i].y = fmaf(p, kv[j][i].y, o[i].y);
        o[i].z = fmaf(p, kv[j][i].z, o[i].z); o[i].w = fmaf(p, kv[j][i].w, o[i].w);
      }
    }
  }
  if (lane == 0) { sm[warp] = m; sl[warp] = l; }
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = (lane + 32 * i) * 4;
    if (c < a.width) *reinterpret_cast<float4*>(rows_o + warp * a.width + c) = o[i];
  }
  __syncthreads();
  const float mx = fmaxf(fmaxf(sm[0], sm[1]), fmaxf(sm[2], sm[3]));
  float w[4], total = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    w[i] = sm[i] == -INFINITY ? 0.f : exp2f(sm[i] - mx);
    total += w[i] * sl[i];
  }
  T* out = static_cast<T*>(a.out) + (static_cast<int64_t>(row) * a.heads + head) * a.width;
  for (int c = threadIdx.x; c < a.width; c += 128)
    out[c] = act_from_f<T>((w[0] * rows_o[c] + w[1] * rows_o[a.width + c] + w[2] * rows_o[2 * a.width + c] + w[3] * rows_o[3 * a.width + c]) / total);
}

template <int WIDTH> static int latent_tc_launch(const LatentArgs& a, cudaStream_t st);      // latent_attention_tc.cu

template <typename T>
static int launch_latent_rows(const LatentArgs& a, cudaStream_t st) {
  const dim3 grid(a.heads, a.m);
  const size_t smem = 4 * sizeof(float) * a.width;
  if (a.width <= 128) return mdb_launch(latent_attn_rows_kernel<T, 1>, grid, dim3(128), smem, st, a);
  if (a.width <= 256) return mdb_launch(latent_attn_rows_kernel<T, 2>, grid, dim3(128), smem, st, a);
  if (a.width <= 512) return mdb_launch(latent_attn_rows_kernel<T, 4>, grid, dim3(128), smem, st, a);
  if (a.width <= 1024) return mdb_launch(latent_attn_rows_kernel<T, 8>, grid, dim3(128), smem, st, a);
  if (a.width <= 2048) return mdb_launch(latent_attn_rows_kernel<T, 16>, grid, dim3(128), smem, st, a);
  return MDB_ERR_UNSUPPORTED;
}

static bool latent_tc_width(int width) { return width == 128 || width == 256 || width == 384 || width == 512; }

}  // namespace mdb

using namespace mdb;

extern "C" {

int64_t mdb_latent_attn_workspace_bytes(int m, int heads, int width, int nsplit) {
  if (m <= 0 || heads <= 0 || width <= 0 || nsplit <= 1) return 0;
  return static_cast<int64_t>(m) * nsplit * heads * (width + 2) * 4;
}

int mdb_latent_attn(int dtype, const void* q, const void* cache, void* out, const int32_t* block_table, int table_stride,
                    const int32_t* row_seq, const int32_t* row_pos, int m, int heads, int width, int num_pages, float scale,
                    int nsplit, void* workspace, int64_t workspace_bytes, mdb_stream_t stream) {
  MDB_REQUIRE(m >= 0 && heads > 0 && width > 0 && num_pages > 0 && table_stride > 0 && nsplit >= 1, MDB_ERR_ARG);
  if (m == 0) return MDB_OK;
  MDB_REQUIRE(q && cache && out && block_table && row_seq && row_pos, MDB_ERR_ARG);
  MDB_REQUIRE(width % 8 == 0 && mdb_aligned16(q) && mdb_aligned16(cache) && mdb_aligned16(out) && mdb_aligned16(workspace), MDB_ERR_ALIGN);
  MDB_REQUIRE(m <= 65535, MDB_ERR_UNSUPPORTED);
  LatentArgs a = {};
  a.q = q; a.cache = cache; a.out = out;
  a.table = block_table; a.table_stride = table_stride; a.num_pages = num_pages;
  a.row_seq = row_seq; a.row_pos = row_pos;
  a.m = m; a.heads = heads; a.width = width;
  a.scale_log2 = scale * 1.4426950408889634f;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (dtype == MDB_F32 || !latent_tc_width(width)) {
    a.nsplit = 1;
    return dtype == MDB_F32 ? launch_latent_rows<float>(a, st) : launch_latent_rows<bf16>(a, st);
  }
  a.nsplit = nsplit;
  const int64_t need = mdb_latent_attn_workspace_bytes(m, heads, width, nsplit);
  MDB_REQUIRE(need == 0 || (workspace != nullptr && workspace_bytes >= need), MDB_ERR_WORKSPACE);
  a.part_o = static_cast<float*>(workspace);
  a.part_ml = a.part_o ? reinterpret_cast<float2*>(a.part_o + static_cast<int64_t>(m) * nsplit * heads * width) : nullptr;
  switch (width) {
    case 128: return latent_tc_launch<128>(a, st);
    case 256: return latent_tc_launch<256>(a, st);
    case 384: return latent_tc_launch<384>(a, st);
    default: return latent_tc_launch<512>(a, st);
  }
}

}  // extern "C"
