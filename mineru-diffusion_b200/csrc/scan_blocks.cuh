// Scans of long prompt portions of few sequences in blocks of 16 tokens, still in fp32 FMAs (included by recurrent.cu, inside its
// namespace, which has the rule for when).
//
// With G_t the product of the decays of a block's tokens 1 .. t (per key channel in the delta rule, one number per head in the
// other recurrences) and S the state in front of the block,
//   u_t = beta_t (v_t - (G_t k_t) S - sum_{j<t} L_tj u_j),      L_tj = k_t . (k_j prod_{j<s<=t} g_s)
//   o_t = (G_t q_t) S + sum_{j<=t} M_tj u_j,                    M_tj = q_t . (k_j prod_{j<s<=t} g_s)
//   S  <- G_16 S + sum_j (k_j prod_{s>j} g_s) u_j^T
// (other recurrences: u_t = b_t v_t, no L).  Every factor is a product of decays, never a quotient, so nothing can overflow and a
// decay of zero is a zero.  A token then costs three FMAs per state element (two without L) and no sum over lanes of its
// own; the token-by-token form spends four (three) and a chain of shuffles for every two tokens.
//
// What bounds it: latency, with few warps per scheduler; a delta rule with 64 columns a CTA by the rate of packed FMAs and shared memory.
// All the states of four prompts of 16 heads are 55 elements per FMA lane of the chip.  A CTA has warps that keep COLS columns of
// the state in registers (CPT columns x 1/16 of the channels a thread: a 16-byte read of shared memory feeds 4 CPT FMAs) and others
// that prepare the next block meanwhile: its operands with cp.async two blocks ahead, the scaled rows, L and M.  Loads stand in
// front of stores: every store might be to what the next load reads, for all the compiler knows, and with a store in each turn of a loop
// the turns come one behind the other (sums of products with the state, u, outputs, scaled rows: 755 -> 665 us for the delta
// rule below); places in memory are worked out once; the mLSTM's normaliser lies in shared memory, a channel per thread.
// The scan alone, 2048 tokens, with those changes: mLSTM, 8 heads of 128 x 256, one, two and four sequences 315 / 350 / 469 -> 250 / 280 /
// 412 us; delta rule, 16 heads of 128 x 128, 463 / 576 / 755 -> 371 / 521 / 640 us.  (Scalar FMAs for the products with the state: 682,
// 444.  The same blocks on tcgen05, operands in three bf16 parts, 128 columns a CTA: 560 and 403, no better for up to 32 sequence heads.)
constexpr int kSbTokens = 16, kSbRing = 3;

template <int MODE, int DP, int COLS, int CPT>
struct SbPlan {
  static constexpr bool DELTA = MODE == kScanDelta;
  static constexpr int ROW = kSbTokens * DP;
  // threads that prepare: L and M of the delta rule, or a block next to few columns, keep eight warps busy
  static constexpr int PREP_THREADS = DELTA || COLS == 16 ? 256 : 128;
  static constexpr int MAIN = COLS / CPT * 16, THREADS = MAIN + PREP_THREADS;      // threads that keep the state; all
  // raw operands, a ring of three blocks: k, q (, g) rows, v, two scalars per token
  static constexpr int RAW_Q = ROW, RAW_G = 2 * ROW, RAW_V = (DELTA ? 3 : 2) * ROW, RAW_S = RAW_V + kSbTokens * COLS, RAW = RAW_S + 2 * kSbTokens;
  // prepared block, two of them: (delta) scaled k and q, k as the update takes it, G_16; L transposed, M; per token four floats
  static constexpr int P_QH = DELTA ? ROW : 0, P_KT = 2 * P_QH, P_G = P_KT + (DELTA ? ROW : 0), P_L = P_G + (DELTA ? DP : 0),
                       P_M = P_L + (DELTA ? 256 : 0), P_T = P_M + 256, PREP = P_T + 4 * kSbTokens;
  static constexpr int OFF_PREP = kSbRing * RAW, OFF_R = OFF_PREP + 2 * PREP, OFF_U = OFF_R + (DELTA ? 2 : 1) * kSbTokens * COLS,
                       OFF_N = OFF_U + 2 * kSbTokens * COLS, FLOATS = OFF_N + DP;
  static constexpr int kSmemBytes = FLOATS * 4;
};

template <int WHICH, int THREADS> __device__ __forceinline__ void sb_bar() { asm volatile("bar.sync %0, %1;" ::"n"(WHICH), "n"(THREADS) : "memory"); }

// Sums 32 values over the 32 lanes: lane l returns the total of value l.
__device__ __forceinline__ float reduce_scatter32(float (&r)[32], int lane) {
#pragma unroll
  for (int o = 16, cur = 16; o > 0; o >>= 1, cur >>= 1) {
    const bool upper = (lane & o) != 0;
#pragma unroll
    for (int j = 0; j < cur; ++j) {
      const float send = upper ? r[j] : r[j + cur], keep = upper ? r[j + cur] : r[j];
      r[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  return r[0];
}

// Sums V values over 16 lanes, the lanes at distance O and less still to come: lane l returns the total of value l * V / (2 O).
template <int V, int O = 8>
__device__ __forceinline__ float sb_reduce16(const float (&r)[V], int l16) {
  if constexpr (O == 0) {
    return r[0];
  } else if constexpr (V == 1) {
    const float h[1] = {r[0] + __shfl_xor_sync(0xffffffffu, r[0], O)};
    return sb_reduce16<1, O / 2>(h, l16);
  } else {
    const bool upper = (l16 & O) != 0;
    float h[V / 2];
#pragma unroll
    for (int j = 0; j < V / 2; ++j) {
      const float send = upper ? r[j] : r[j + V / 2], keep = upper ? r[j + V / 2] : r[j];
      h[j] = keep + __shfl_xor_sync(0xffffffffu, send, O);
    }
    return sb_reduce16<V / 2, O / 2>(h, l16);
  }
}

__device__ __forceinline__ float sum2(f32x2 v) { const float2 x = unpack2(v); return x.x + x.y; }

template <int MODE, int DP, int COLS, int CPT>
__global__ void __launch_bounds__(SbPlan<MODE, DP, COLS, CPT>::THREADS, 1) scan_blocks_kernel(const mdb_scan_args a) {
  using P = SbPlan<MODE, DP, COLS, CPT>;
  constexpr bool DELTA = P::DELTA, MLSTM = MODE == kScanMlstm;
  constexpr int MAIN = P::MAIN, T = kSbTokens, PW = P::PREP_THREADS / 32, PASSES = T / 2 / PW, TPW = T / PW, NR = DP / 64, NP = DP / 64;      // float4 per lane and column; channel pairs per lane of a row
  extern __shared__ __align__(16) float sb_smem[];
  pdl_launch_dependents();
  pdl_wait();
  const ScanJob w = scan_job<MODE, DP, COLS>(a);
  if (!w.live) return;
  const int blocks16 = (w.columns + kScanBlockCols - 1) / kScanBlockCols, block0 = w.col0 / kScanBlockCols;
  float* mstate = MLSTM ? a.mstate + (static_cast<int64_t>(w.slot) * a.heads + w.head) * blocks16 : nullptr;
  const int nblocks = (w.t_end - w.t_begin + T - 1) / T;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* const R = sb_smem + P::OFF_R;      // (delta: k-side, then) q-side products with the state, [token][column]
  float* const U = sb_smem + P::OFF_U;      // u as pairs (u, u), [token][column]

  if (threadIdx.x >= MAIN) {
    // ------------------------------------------------------------------------------------------------ preparing warps
    const int tid = threadIdx.x - MAIN, pw = warp - MAIN / 32;
    const bool v16 = (a.vdim & 3) == 0 && (reinterpret_cast<uintptr_t>(a.v) & 15) == 0;
    // places of a thread's 16-byte pieces, worked out once: KP rows of k, q and g, VP of v
    constexpr int KT = P::PREP_THREADS / (DP / 4), KP = T / KT, VT = P::PREP_THREADS / (COLS / 4), VP = T > VT ? T / VT : 1;
    static_assert(KT <= T && T % KT == 0 && (VT >= T || T % VT == 0), "whole rounds over a block's rows");
    const int ft = tid / (DP / 4), fc = tid % (DP / 4) * 4, vt = tid / (COLS / 4), vc = tid % (COLS / 4) * 4;
    const int64_t kstep = static_cast<int64_t>(a.kv_heads) * DP, gstep = static_cast<int64_t>(a.heads) * DP, vstep = static_cast<int64_t>(a.heads) * a.vdim;
    const int64_t k_at = static_cast<int64_t>(w.kvh) * DP + (w.t_begin + ft) * kstep + fc;
    const float* kp = a.k + k_at;
    const float* qp = a.q + k_at;
    const float* gp = DELTA ? a.g + static_cast<int64_t>(w.head) * DP + (w.t_begin + ft) * gstep + fc : nullptr;
    const float* vp = a.v + static_cast<int64_t>(w.head) * a.vdim + w.col0 + (w.t_begin + vt) * vstep + vc;
    const bool v_whole = v16 && w.col0 + vc < a.vdim;
    auto fetch = [&](int b) {                                   // blocks one after the other
      if (b < nblocks) {
        const int t0 = w.t_begin + b * T, n = min(T, w.t_end - t0);
        float* st = sb_smem + (b % kSbRing) * P::RAW;
        const uint32_t base = smem_u32(st);
#pragma unroll
        for (int i = 0; i < KP; ++i) {
          const int t = ft + i * KT;
          if (t < n) {
            cp_async16(base + (t * DP + fc) * 4, kp + i * KT * kstep);
            cp_async16(base + (P::RAW_Q + t * DP + fc) * 4, qp + i * KT * kstep);
            if (DELTA) cp_async16(base + (P::RAW_G + t * DP + fc) * 4, gp + i * KT * gstep);
          } else {      // tokens behind the portion: no key, no query, no decay
            *reinterpret_cast<float4*>(st + t * DP + fc) = make_float4(0.f, 0.f, 0.f, 0.f);
            *reinterpret_cast<float4*>(st + P::RAW_Q + t * DP + fc) = make_float4(0.f, 0.f, 0.f, 0.f);
            if (DELTA) *reinterpret_cast<float4*>(st + P::RAW_G + t * DP + fc) = make_float4(1.f, 1.f, 1.f, 1.f);
          }
        }
#pragma unroll
        for (int i = 0; i < VP; ++i) {
          const int t = vt + i * VT;
          if (t >= T) break;
          float* vs = st + P::RAW_V + t * COLS + vc;
          const float* from = vp + i * VT * vstep;
          if (v_whole && t < n) {
            cp_async16(smem_u32(vs), from);
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              if (t < n && w.col0 + vc + e < a.vdim) cp_async4(smem_u32(vs + e), from + e);
              else vs[e] = 0.f;
            }
          }
        }
        kp += T * kstep;
        qp += T * kstep;
        gp += T * gstep;
        vp += T * vstep;
        if (tid < T) {
          const int64_t th = static_cast<int64_t>(t0 + tid) * a.heads + w.head;
          if (tid < n) {
            if (DELTA) {
              cp_async4(base + (P::RAW_S + 2 * tid) * 4, a.scalars + 4 * th + 3);
            } else {
              cp_async4(base + (P::RAW_S + 2 * tid) * 4, a.s0 + th);
              cp_async4(base + (P::RAW_S + 2 * tid + 1) * 4, a.s1 + th);
            }
          } else {
            // delta: no correction; mLSTM: input gate shut, forget gate open; decay scan: no decay, no step
            st[P::RAW_S + 2 * tid] = DELTA ? 0.f : (MLSTM ? -INFINITY : 1.f);
            st[P::RAW_S + 2 * tid + 1] = 0.f;
          }
        }
      }
      cp_async_commit();
    };

    float run_max = MLSTM && !w.fresh ? mstate[block0] : 0.f;
    // the normaliser, one more column of the mLSTM's state: only the CTA of the first columns has it, a channel per thread
    const bool norm = MLSTM && w.col0 == 0;
    float* const nrm = sb_smem + P::OFF_N;
    static_assert(!MLSTM || P::PREP_THREADS >= DP, "a thread per channel of the normaliser");
    if (norm && tid < DP) nrm[tid] = w.fresh ? 0.f : w.state[static_cast<int64_t>(a.vdim) * DP + tid];
    // lane's share of a row: NP channel pairs
    auto row_pairs = [&](const float* row, f32x2 (&x)[NP]) {
      if (NP == 2) {
        lds2(row + lane * 4, x[0], x[NP - 1]);
      } else {
        x[0] = *reinterpret_cast<const f32x2*>(row + lane * 2);
      }
    };

    auto prepare = [&](int b) {
      const float* raw = sb_smem + (b % kSbRing) * P::RAW;
      float* prep = sb_smem + P::OFF_PREP + (b & 1) * P::PREP;
      float4* per_token = reinterpret_cast<float4*>(prep + P::P_T);
      if (DELTA) {
        if (tid < DP) {
          const int c = tid;
          float kk[T], gg[T], qq[T], acc = 1.f;
#pragma unroll
          for (int t = 0; t < T; ++t) {
            kk[t] = raw[t * DP + c];
            gg[t] = raw[P::RAW_G + t * DP + c];
            qq[t] = raw[P::RAW_Q + t * DP + c];
          }
#pragma unroll
          for (int t = 0; t < T; ++t) {
            acc *= gg[t];
            prep[t * DP + c] = acc * kk[t];
            prep[P::P_QH + t * DP + c] = acc * qq[t];
          }
          prep[P::P_G + c] = acc;
          acc = 1.f;
#pragma unroll
          for (int t = T - 1; t >= 0; --t) {
            prep[P::P_KT + t * DP + c] = acc * kk[t];
            acc *= gg[t];
          }
        }
        if (tid < T) per_token[tid].x = raw[P::RAW_S + 2 * tid];      // beta
        // L and M: a warp takes two neighbouring keys; the first warps, who also scale the rows, those with few tokens behind them
        static_assert(!DELTA || PASSES == 1, "a pair of keys per warp");
        const int j0 = pw >= 4 ? 2 * (pw - 4) : T - 2 - 2 * pw;
        {
          f32x2 p[2][NP];
          float acc[2][32];
#pragma unroll
          for (int i = 0; i < NP; ++i) p[0][i] = p[1][i] = 0ull;
          // A branch for AT tokens at a time, whose loads go out together: four next to 16 or 32 columns, one next to 64, where the
          // other warps want the issue slots (4 x 2048 tokens 640 against 664 us; 2 x 2048, 32 columns, 539 against 521; 1 x 2048, 16
          // columns, 383 against 371).
          constexpr int AT = COLS == 64 ? 1 : 4;
#pragma unroll
          for (int t0 = 0; t0 < T; t0 += AT) {
            if (t0 + AT - 1 < j0) {
#pragma unroll
              for (int i = 0; i < 2 * AT; ++i) acc[0][2 * t0 + i] = acc[1][2 * t0 + i] = 0.f;
              continue;
            }
            f32x2 k[AT][NP], q[AT][NP], g[AT][NP];
#pragma unroll
            for (int e = 0; e < AT; ++e) {
              row_pairs(raw + (t0 + e) * DP, k[e]);
              row_pairs(raw + P::RAW_Q + (t0 + e) * DP, q[e]);
              row_pairs(raw + P::RAW_G + (t0 + e) * DP, g[e]);
            }
#pragma unroll
            for (int e = 0; e < AT; ++e) {
              const int t = t0 + e;
#pragma unroll
              for (int jj = 0; jj < 2; ++jj) {
                f32x2 l = 0ull, m = 0ull;
#pragma unroll
                for (int i = 0; i < NP; ++i) {
                  p[jj][i] = t == j0 + jj ? k[e][i] : mul2(p[jj][i], g[e][i]);      // nothing in front of the key itself
                  l = fma2(p[jj][i], k[e][i], l);
                  m = fma2(p[jj][i], q[e][i], m);
                }
                acc[jj][2 * t] = sum2(l);
                acc[jj][2 * t + 1] = sum2(m);
              }
            }
          }
#pragma unroll
          for (int jj = 0; jj < 2; ++jj) {
            const float total = reduce_scatter32(acc[jj], lane);
            const int t = lane >> 1, j = j0 + jj;
            if (lane & 1) prep[P::P_M + t * T + j] = total;
            else prep[P::P_L + j * T + t] = raw[P::RAW_S + 2 * t] * total;      // beta_t L_tj
          }
        }
      } else {
        // gates of the block: forget and input factor per token, in the mLSTM relative to the running maximum
        float fa = 1.f, fb = 0.f, em = 0.f;
        {
          const int l = lane & 15;
          const float s0 = raw[P::RAW_S + 2 * l], s1 = raw[P::RAW_S + 2 * l + 1];
          if (MLSTM) {
            // m_t = max(f_t + m_(t-1), i_t) as a scan of the maps x -> max(x + F, I); tokens behind the portion keep m
            float F = s1, I = s0;
#pragma unroll
            for (int o = 1; o < T; o <<= 1) {
              const float Fp = __shfl_up_sync(0xffffffffu, F, o, 16), Ip = __shfl_up_sync(0xffffffffu, I, o, 16);
              if (l >= o) { I = fmaxf(Ip + F, I); F += Fp; }
            }
            const float m = fmaxf(F + run_max, I);
            float mp = __shfl_up_sync(0xffffffffu, m, 1, 16);
            if (l == 0) mp = run_max;
            fa = expf(s1 + mp - m);
            fb = expf(s0 - m);
            em = expf(-m);
            run_max = __shfl_sync(0xffffffffu, m, T - 1);
          } else {
            fa = s0;
            fb = s1;
          }
        }
        // every lane: product of the forget factors of tokens 0 .. t, of those behind t, of those behind j up to t
        const int t = lane & 15, jl = lane >> 4;
        float head = 1.f, tail = 1.f;
        // the two keys a warp takes in a pass: from either end, so that the tokens behind them even out
        auto first_key = [&](int pass) { return pass ? T - 2 - 2 * pw : 2 * pw; };
        float between[PASSES];
#pragma unroll
        for (int pass = 0; pass < PASSES; ++pass) between[pass] = 1.f;
#pragma unroll
        for (int s = 0; s < T; ++s) {
          const float f = __shfl_sync(0xffffffffu, fa, s);
          if (s <= t) head *= f;
          if (s > t) tail *= f;
#pragma unroll
          for (int pass = 0; pass < PASSES; ++pass)
            if (s > first_key(pass) + jl && s <= t) between[pass] *= f;
        }
        if (pw == 0 && lane < T) per_token[lane] = make_float4(head, fb * tail, em, 0.f);
#pragma unroll
        for (int pass = 0; pass < PASSES; ++pass) {
          const int j0 = first_key(pass), j = j0 + jl;
          float acc[32];
          f32x2 k[2][NP];
          row_pairs(raw + j0 * DP, k[0]);
          row_pairs(raw + (j0 + 1) * DP, k[1]);
#pragma unroll
          for (int t2 = 0; t2 < T; ++t2) {
            acc[t2] = acc[T + t2] = 0.f;
            if (t2 < j0) continue;
            f32x2 q[NP];
            row_pairs(raw + P::RAW_Q + t2 * DP, q);
#pragma unroll
            for (int jj = 0; jj < 2; ++jj) {
              f32x2 s = 0ull;
#pragma unroll
              for (int i = 0; i < NP; ++i) s = fma2(k[jj][i], q[i], s);
              acc[jj * T + t2] = sum2(s);
            }
          }
          const float total = reduce_scatter32(acc, lane);      // q_t . k_j, t = lane & 15, j = j0 + lane / 16
          const float bj = __shfl_sync(0xffffffffu, fb, j);
          prep[P::P_M + t * T + j] = j <= t ? between[pass] * bj * total : 0.f;
        }
        if (norm) {
          // q_t . n for a warp's tokens; when all have read it n moves past the block
          float mine = 0.f;
          f32x2 nv[NP];
          row_pairs(nrm, nv);
#pragma unroll
          for (int i2 = 0; i2 < TPW; ++i2) {
            f32x2 q[NP], s = 0ull;
            row_pairs(raw + P::RAW_Q + (TPW * pw + i2) * DP, q);
#pragma unroll
            for (int i = 0; i < NP; ++i) s = fma2(nv[i], q[i], s);
            const float qn = warp_sum(sum2(s));
            if (lane == i2) mine = qn;
          }
          sb_bar<2, P::PREP_THREADS>();                                        // and M is whole
          if (tid < DP) {
            float n = nrm[tid] * per_token[T - 1].x;
#pragma unroll
            for (int s = 0; s < T; ++s) n = fmaf(raw[s * DP + tid], per_token[s].y, n);
            nrm[tid] = n;
          }
          if (lane < TPW) {
            const int tt = TPW * pw + lane, tok = w.t_begin + b * T + tt;
            const float4 pt = per_token[tt];
            float s = 0.f;
#pragma unroll
            for (int j = 0; j < T; ++j) s += prep[P::P_M + tt * T + j];
            if (tok < w.t_end) a.den[static_cast<int64_t>(tok) * a.heads + w.head] = fmaxf(fabsf(fmaf(pt.x, mine, s)), pt.z) + 1e-6f;
          }
        }
      }
    };

    fetch(0);
    fetch(1);
    cp_async_wait<1>();
    sb_bar<2, P::PREP_THREADS>();
    prepare(0);
    __syncthreads();
    for (int b = 0; b < nblocks; ++b) {
      fetch(b + 2);                     // its place was read for the last time before the barrier
      if (b + 1 < nblocks) {
        cp_async_wait<1>();
        sb_bar<2, P::PREP_THREADS>();
        prepare(b + 1);
      }
      __syncthreads();
    }
    cp_async_wait<0>();
    if (norm && tid < DP) w.state[static_cast<int64_t>(a.vdim) * DP + tid] = nrm[tid];
    if (MLSTM && tid == 0) {
      // the copies of the running maximum of this CTA's columns; the normaliser's belongs to the first CTA
      for (int i = block0; i < blocks16 && i * kScanBlockCols < w.col0 + COLS && i * kScanBlockCols < a.vdim; ++i) mstate[i] = run_max;
      if (norm && a.vdim % kScanBlockCols == 0) mstate[blocks16 - 1] = run_max;
    }
    return;
  }

  // ---------------------------------------------------------------------------------------------------- state warps
  const int l16 = threadIdx.x & 15, cg = threadIdx.x >> 4, col = cg * CPT, mycol = w.col0 + col;
  const float skip = MODE == kScanDecay && a.skip != nullptr ? a.skip[w.head] : 0.f;
  f32x2 S[CPT][2 * NR];
#pragma unroll
  for (int i = 0; i < CPT; ++i)
#pragma unroll
    for (int c = 0; c < NR; ++c) {
      float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
      if (!w.fresh && mycol + i < a.vdim)
        x = *reinterpret_cast<const float4*>(w.state + static_cast<int64_t>(mycol + i) * DP + c * 64 + l16 * 4);
      S[i][2 * c] = pack2(x.x, x.y);
      S[i][2 * c + 1] = pack2(x.z, x.w);
    }
  __syncthreads();
  for (int b = 0; b < nblocks; ++b) {
    const float* raw = sb_smem + (b % kSbRing) * P::RAW;
    const float* prep = sb_smem + P::OFF_PREP + (b & 1) * P::PREP;
    const float4* per_token = reinterpret_cast<const float4*>(prep + P::P_T);
    // products with the state in front of the block: of a token's k and q (delta), or of two tokens' q, per exchange
    constexpr int ROWS = DELTA ? 2 * T : T;
    float totals[ROWS / 2];
#pragma unroll
    for (int r = 0; r < ROWS; r += 2) {
      const float* x0 = DELTA ? prep + (r >> 1) * DP + l16 * 4 : raw + P::RAW_Q + r * DP + l16 * 4;
      const float* x1 = DELTA ? prep + P::P_QH + (r >> 1) * DP + l16 * 4 : x0 + DP;
      f32x2 acc[2][CPT];
#pragma unroll
      for (int i = 0; i < CPT; ++i) acc[0][i] = acc[1][i] = 0ull;
#pragma unroll
      for (int c = 0; c < NR; ++c) {
        f32x2 y0[2], y1[2];
        lds2(x0 + c * 64, y0[0], y0[1]);
        lds2(x1 + c * 64, y1[0], y1[1]);
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int i = 0; i < CPT; ++i) {
            acc[0][i] = fma2(S[i][2 * c + e], y0[e], acc[0][i]);
            acc[1][i] = fma2(S[i][2 * c + e], y1[e], acc[1][i]);
          }
      }
      float v[2 * CPT];
#pragma unroll
      for (int i = 0; i < CPT; ++i) {
        v[i] = sum2(acc[0][i]);
        v[CPT + i] = sum2(acc[1][i]);
      }
      totals[r / 2] = sb_reduce16<2 * CPT>(v, l16);
    }
    {
      constexpr int PER = 16 / (2 * CPT);                // lanes that hold the same sum
      const int at = l16 / PER, which = at / CPT, i = at % CPT;
      if (l16 % PER == 0) {
#pragma unroll
        for (int r = 0; r < ROWS; r += 2) R[DELTA ? (which * T + (r >> 1)) * COLS + col + i : (r + which) * COLS + col + i] = totals[r / 2];
      }
    }
    if (!DELTA) {
      constexpr int N = (T * COLS + MAIN - 1) / MAIN;
      float u[N];
#pragma unroll
      for (int n = 0; n < N; ++n) {
        const int i = min(static_cast<int>(threadIdx.x) + n * MAIN, T * COLS - 1);
        u[n] = raw[P::RAW_V + i] * per_token[i / COLS].y;
      }
#pragma unroll
      for (int n = 0; n < N; ++n)
        if (threadIdx.x + n * MAIN < T * COLS) *reinterpret_cast<float2*>(U + 2 * (threadIdx.x + n * MAIN)) = make_float2(u[n], u[n]);
    }
    sb_bar<1, MAIN>();
    if (DELTA) {
      if (threadIdx.x < COLS) {
        float u[T];
#pragma unroll
        for (int t = 0; t < T; ++t) u[t] = per_token[t].x * (raw[P::RAW_V + t * COLS + threadIdx.x] - R[t * COLS + threadIdx.x]);
#pragma unroll
        for (int j = 0; j < T; ++j) {
          float l[T];
#pragma unroll
          for (int c = j / 4; c < T / 4; ++c) *reinterpret_cast<float4*>(l + 4 * c) = *reinterpret_cast<const float4*>(prep + P::P_L + j * T + 4 * c);
#pragma unroll
          for (int t = j + 1; t < T; ++t) u[t] = fmaf(-l[t], u[j], u[t]);
        }
#pragma unroll
        for (int j = 0; j < T; ++j) *reinterpret_cast<float2*>(U + 2 * (j * COLS + threadIdx.x)) = make_float2(u[j], u[j]);
      }
      sb_bar<1, MAIN>();
    }
    // the state moves past the block
    const float* kt = (DELTA ? prep + P::P_KT : raw) + l16 * 4;
    if (DELTA) {
#pragma unroll
      for (int c = 0; c < NR; ++c) {
        f32x2 g[2];
        lds2(prep + P::P_G + l16 * 4 + c * 64, g[0], g[1]);
#pragma unroll
        for (int i = 0; i < CPT; ++i) {
          S[i][2 * c] = mul2(S[i][2 * c], g[0]);
          S[i][2 * c + 1] = mul2(S[i][2 * c + 1], g[1]);
        }
      }
    } else {
      const float whole = per_token[T - 1].x;
      const f32x2 g = pack2(whole, whole);
#pragma unroll
      for (int i = 0; i < CPT; ++i)
#pragma unroll
        for (int c = 0; c < 2 * NR; ++c) S[i][c] = mul2(S[i][c], g);
    }
#pragma unroll 8
    for (int t = 0; t < T; ++t) {
      f32x2 u[CPT];
#pragma unroll
      for (int i = 0; i < CPT; i += 2) lds2(U + 2 * (t * COLS + col + i), u[i], u[i + 1]);
#pragma unroll
      for (int c = 0; c < NR; ++c) {
        f32x2 k[2];
        lds2(kt + t * DP + c * 64, k[0], k[1]);
#pragma unroll
        for (int i = 0; i < CPT; ++i) {
          S[i][2 * c] = fma2(k[0], u[i], S[i][2 * c]);
          S[i][2 * c + 1] = fma2(k[1], u[i], S[i][2 * c + 1]);
        }
      }
    }
    // outputs: a thread takes every (MAIN / COLS)-th token of a column
    {
      constexpr int STEP = MAIN / COLS;
      const int c = threadIdx.x % COLS, first = threadIdx.x / COLS;
      float x[T];
#pragma unroll
      for (int j = 0; j < T; ++j) x[j] = DELTA ? U[2 * (j * COLS + c)] : raw[P::RAW_V + j * COLS + c];
      constexpr int N = T / STEP;
      float out[N];
#pragma unroll
      for (int n = 0; n < N; ++n) {
        const int t = first + n * STEP;
        float m[T], o = DELTA ? R[(T + t) * COLS + c] : R[t * COLS + c] * per_token[t].x;
#pragma unroll
        for (int j = 0; j < T; j += 4) *reinterpret_cast<float4*>(m + j) = *reinterpret_cast<const float4*>(prep + P::P_M + t * T + j);
#pragma unroll
        for (int j = 0; j < T; ++j)
          if (j <= t) o = fmaf(m[j], x[j], o);      // not behind t, where a value may be anything
        if (MODE == kScanDecay) o = fmaf(skip, raw[P::RAW_V + t * COLS + c], o);
        out[n] = o;
      }
#pragma unroll
      for (int n = 0; n < N; ++n) {
        const int tok = w.t_begin + b * T + first + n * STEP;
        if (tok < w.t_end && w.col0 + c < a.vdim) a.out[(static_cast<int64_t>(tok) * a.heads + w.head) * a.vdim + w.col0 + c] = out[n];
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < CPT; ++i)
    if (mycol + i < a.vdim) {
#pragma unroll
      for (int c = 0; c < NR; ++c) {
        const float2 lo = unpack2(S[i][2 * c]), hi = unpack2(S[i][2 * c + 1]);
        *reinterpret_cast<float4*>(w.state + static_cast<int64_t>(mycol + i) * DP + c * 64 + l16 * 4) = make_float4(lo.x, lo.y, hi.x, hi.y);
      }
    }
}

template <int MODE, int DP, int COLS, int CPT>
int launch_scan_blocks(const mdb_scan_args& a, cudaStream_t st) {
  using P = SbPlan<MODE, DP, COLS, CPT>;
  static_assert(P::kSmemBytes <= 227 * 1024, "shared memory of the scan in blocks");
  auto kernel = scan_blocks_kernel<MODE, DP, COLS, CPT>;
  static PerDeviceOnce attr_once;
  const int dev = attr_once.slot();
  if (dev < 0) return MDB_ERR_CUDA;
  if (!attr_once.done[dev]) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, P::kSmemBytes) != cudaSuccess) return MDB_ERR_CUDA;
    attr_once.done[dev] = true;
  }
  return mdb_launch(kernel, dim3((a.vdim + COLS - 1) / COLS, a.heads, a.bs), dim3(P::THREADS), P::kSmemBytes, st, a);
}
