// Causal attention over cached latents: every query head of a token reads the same latent row of a key, which stands
// for its key and its value alike (the per-head key projection is folded into the query, the per-head value
// projection follows the attention), so a key costs one latent row of memory traffic for all heads.
//
//   latent_attn_tc_kernel    bf16, widths of 128 to 512 (latent_attention_tc.cu); parts of a context are merged by
//                            latent_combine_kernel.
//   latent_attn_rows_kernel  fp32, and widths the first kernel does not take: one CTA per token and one to four heads, a
//                            warp per key.
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

// The sums over a warp's lanes of N values at once: lane v * 32 / N (and those up to the next) has value v.  The lanes' tree is the
// same for every N.
template <int N>
__device__ __forceinline__ float lanes_sum(float (&v)[N], int lane) {
  int bit = 16;
#pragma unroll
  for (int n = N / 2; n >= 1; n /= 2, bit /= 2) {
    const bool up = lane & bit;
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const float send = up ? v[i] : v[i + n];
      v[i] = (up ? v[i + n] : v[i]) + __shfl_xor_sync(~0u, send, bit);
    }
  }
  for (; bit >= 1; bit /= 2) v[0] += __shfl_xor_sync(~0u, v[0], bit);
  return v[0];
}

// One CTA of four warps per (row, HEADS heads); warp w takes keys w, w + 4, ...; a lane owns every 32nd float4 group of four
// channels.  NV = channels per lane / 4.  Several keys at a time, as registers allow: their rows are in flight together and share a
// new maximum, and a lane works out the weight of one (head, key).  A head's bits do not depend on HEADS.
// The longest contexts of a prompt, its last rows, go first.
// What bounds it: few rows, the latency of a step (a row's place, its loads, the sums, the weights); many, issue slots (16 packed FMAs
// and about 6 other instructions for a head's key of 256 channels).  500 rows of 8 heads, width 256, a prompt: one head at a time with a
// sum and a weight per lane and key 112 us, out of L2; HEADS 1, 2, 4: 76, 57, 50.
template <typename T, int NV, int HEADS>
__global__ void __launch_bounds__(128) latent_attn_rows_kernel(const LatentArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int KEYS = NV <= 2 ? 4 : NV <= 4 ? 2 : 1, N = HEADS * KEYS, STEP = 32 / N;
  __shared__ float sm[4][HEADS], sl[4][HEADS];
  extern __shared__ float rows_o[];        // [4][HEADS][width]
  const int row = a.m - 1 - blockIdx.y, head0 = blockIdx.x * HEADS, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int pos = a.row_pos[row];
  if (pos < 0) return;
  const int32_t* table = a.table + static_cast<int64_t>(a.row_seq[row]) * a.table_stride;
  f32x2 qv[HEADS][NV][2], o[HEADS][NV][2];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = (lane + 32 * i) * 4;
#pragma unroll
    for (int h = 0; h < HEADS; ++h) {
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (c < a.width) v = act_load4(static_cast<const T*>(a.q) + (static_cast<int64_t>(row) * a.heads + min(head0 + h, a.heads - 1)) * a.width + c);
      qv[h][i][0] = pack2(v.x, v.y);
      qv[h][i][1] = pack2(v.z, v.w);
      o[h][i][0] = o[h][i][1] = pack2(0.f, 0.f);
    }
  }
  const int mine = lane / STEP % KEYS;      // the key, of the KEYS of a step, whose weight this lane works out
  float m = -INFINITY, l = 0.f;
  for (int key = warp; key <= pos; key += 4 * KEYS) {
    f32x2 kv[KEYS][NV][2];
#pragma unroll
    for (int j = 0; j < KEYS; ++j) {
      const T* kr = static_cast<const T*>(a.cache) + latent_slot(a, table, min(key + 4 * j, pos)) * a.width;
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const int c = (lane + 32 * i) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (c < a.width) v = act_load4(kr + c);
        kv[j][i][0] = pack2(v.x, v.y);
        kv[j][i][1] = pack2(v.z, v.w);
      }
    }
    float s[N];
#pragma unroll
    for (int h = 0; h < HEADS; ++h)
#pragma unroll
      for (int j = 0; j < KEYS; ++j) {
        f32x2 t = pack2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < NV; ++i) {
          t = fma2(qv[h][i][0], kv[j][i][0], t);
          t = fma2(qv[h][i][1], kv[j][i][1], t);
        }
        const float2 u = unpack2(t);
        s[h * KEYS + j] = u.x + u.y;
      }
    float w = lanes_sum<N>(s, lane) * a.scale_log2;
    w = key + 4 * mine <= pos ? w : -INFINITY;
    float m_new = w;
#pragma unroll
    for (int b = STEP; b < STEP * KEYS; b *= 2) m_new = fmaxf(m_new, __shfl_xor_sync(~0u, m_new, b));
    m_new = fmaxf(m_new, m);
    const float f = exp2f(m - m_new);
    m = m_new;
    w = exp2f(w - m);
    l = l * f + w;
#pragma unroll
    for (int h = 0; h < HEADS; ++h) {
      const float fs = N == 1 ? f : __shfl_sync(~0u, f, h * KEYS * STEP);
      const f32x2 fh = pack2(fs, fs);
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        o[h][i][0] = mul2(o[h][i][0], fh);
        o[h][i][1] = mul2(o[h][i][1], fh);
      }
#pragma unroll
      for (int j = 0; j < KEYS; ++j) {
        const float ps = N == 1 ? w : __shfl_sync(~0u, w, (h * KEYS + j) * STEP);
        const f32x2 p = pack2(ps, ps);
#pragma unroll
        for (int i = 0; i < NV; ++i) {
          o[h][i][0] = fma2(p, kv[j][i][0], o[h][i][0]);
          o[h][i][1] = fma2(p, kv[j][i][1], o[h][i][1]);
        }
      }
    }
  }
#pragma unroll
  for (int b = STEP; b < STEP * KEYS; b *= 2) l += __shfl_xor_sync(~0u, l, b);
  if (lane % (STEP * KEYS) == 0) { sm[warp][lane / (STEP * KEYS)] = m; sl[warp][lane / (STEP * KEYS)] = l; }
#pragma unroll
  for (int h = 0; h < HEADS; ++h)
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = (lane + 32 * i) * 4;
      const float2 lo = unpack2(o[h][i][0]), hi = unpack2(o[h][i][1]);
      if (c < a.width) *reinterpret_cast<float4*>(rows_o + (warp * HEADS + h) * a.width + c) = make_float4(lo.x, lo.y, hi.x, hi.y);
    }
  __syncthreads();
  T* out = static_cast<T*>(a.out) + (static_cast<int64_t>(row) * a.heads + head0) * a.width;
#pragma unroll
  for (int h = 0; h < HEADS; ++h) {
    if (head0 + h >= a.heads) break;
    const float mx = fmaxf(fmaxf(sm[0][h], sm[1][h]), fmaxf(sm[2][h], sm[3][h]));
    float w[4], total = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      w[i] = sm[i][h] == -INFINITY ? 0.f : exp2f(sm[i][h] - mx);
      total += w[i] * sl[i][h];
    }
    const float* ro = rows_o + h * a.width;
    const int part = HEADS * a.width;
    for (int c = threadIdx.x; c < a.width; c += 128)
      out[h * a.width + c] = act_from_f<T>((w[0] * ro[c] + w[1] * ro[part + c] + w[2] * ro[2 * part + c] + w[3] * ro[3 * part + c]) / total);
  }
}

template <int WIDTH> static int latent_tc_launch(const LatentArgs& a, cudaStream_t st);      // latent_attention_tc.cu

template <typename T, int NV, int HEADS>
static int latent_rows_form(const LatentArgs& a, cudaStream_t st) {
  return mdb_launch(latent_attn_rows_kernel<T, NV, HEADS>, dim3((a.heads + HEADS - 1) / HEADS, a.m), dim3(128),
                    4 * sizeof(float) * HEADS * a.width, st, a);
}

// How many heads share the reading of a key: as many as leave the chip full (heads of 256 channels, us with 1, 2, 4 of them; two where
// that leaves an SM a CTA, four where it leaves three).
//   prompt of 500 rows, 8 heads   76   57   50        64 rows behind 3000 keys, 16 heads   233  228  250
//   prompt of 250, 16 heads       42   32   30        128 behind 2000, 16 heads            296  266  272
//   prompt of 137, 8 heads        12   12   12        8 behind 2000, 8 heads                83   87  103
// Heads of 512 channels: 300 rows of 16 heads, a prompt, 100, 86, 77; 40 rows behind 2000 keys 232, 241, 282: two are never the best by
// much.  Behind 512 channels registers leave no room for a second head (200 rows of 16 heads of 640 channels 90, 101).
template <typename T, int NV>
static int latent_rows_few(const LatentArgs& a, cudaStream_t st) {
  const int64_t sms = at_sm_count(), m = a.m;
  if (m * (a.heads / 4) >= 3 * sms) return latent_rows_form<T, NV, 4>(a, st);
  if constexpr (NV < 4) {
    if (m * (a.heads / 2) >= sms) return latent_rows_form<T, NV, 2>(a, st);
  }
  return latent_rows_form<T, NV, 1>(a, st);
}

template <typename T>
static int launch_latent_rows(const LatentArgs& a, cudaStream_t st) {
  if (a.width <= 128) return latent_rows_few<T, 1>(a, st);
  if (a.width <= 256) return latent_rows_few<T, 2>(a, st);
  if (a.width <= 512) return latent_rows_few<T, 4>(a, st);
  if (a.width <= 1024) return latent_rows_form<T, 8, 1>(a, st);
  if (a.width <= 2048) return latent_rows_form<T, 16, 1>(a, st);
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
