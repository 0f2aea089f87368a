// Gated delta rule (linear attention of Qwen3-Next / Kimi-style GDN blocks), recurrent over groups of tokens:
//
//   S  <- exp(g_t) * S                         decay            S: [Dk, Dv] per (sequence, value head), fp32
//   u  <- beta_t (v_t - S^T k_t)               delta            u: [Dv]
//   S  <- S + k_t u^T
//   o_t = S^T (scale * q_t)
//
// bf16 prompts go by chunks of 16 tokens on the tensor cores (further down, the chunked form of Yang et al., "Gated Delta
// Networks: Improving Mamba2 with Delta Rule", 2024); decode rows and other short sequences a token at a
// time (gdn_step_kernel), and so does everything where results must not depend on what else is in a step or on where a prompt is cut;
// fp16 prompts by groups of G = 4 on the fp32 units, as follows.  With S as it is before the group, G_t the sum of g over the group's
// tokens up to t and D_tj = exp(G_t - G_j) (never above 1):
//
//   u_t = beta_t (v_t - exp(G_t) k_t . S - sum_{j<t} D_tj (k_t . k_j) u_j)
//   o_t = scale (exp(G_t) q_t . S + sum_{j<=t} D_tj (q_t . k_j) u_j)
//   S  <- exp(G_last) S + sum_j k_j D_last,j u_j^T
//
// so the 2 G products with S are formed in one pass over it, lanes exchange sums once per group and S is rewritten once.
// The products among q and k of a group and their lengths come from a small kernel in front, once per key head; the lengths
// scale the sums, so the rows themselves are used as they are.  All of it in fp32.
//
// One CTA = one (sequence, value head, 32 value columns): columns are independent of one another.  16 lanes share 4 columns;
// lane r holds rows r*4 + 64 i of them, pairs of rows packed for the two-wide fp32 instructions.  Of a group's 8 x 4 partial
// sums, halving exchanges leave one column's four per lane.  Tokens are staged 16 at a time as fp32 rows, the next 16 on their
// way in registers meanwhile.  What bounds it: for prompts the fp32 units (13 multiply-adds per state element and 4 tokens); for
// decode steps the state's read and write.
// 4 prompts of 3949 tokens in all (the longest 2048), 32 heads: 3382 us with a token at a time and a thread per column,
// 705 us by groups, 313 us by chunks.  64 decode rows: 58.6 us, now 49.5 us.
// The state is read from / written to a slot pool, so that decode steps and chunked prefill continue where the last call stopped.
// Covers ChunkGatedDeltaRule.forward (vllm_metax/registry/custom_ops/layers/mamba/qwen_gdn_linear_attn.py:16-88)
// and the fused recurrent decode step of the same block.
#include <type_traits>

#include "common.cuh"
#include "attn_decode.cuh"
#include "f32x2.cuh"
#include "ops.h"
#include "pdl.cuh"

namespace b200 {

// What a token's products need: 1 / |k|, scale / |q|, k_t . k_{t-d} (d = 1..3), q_t . k_{t-d} (d = 0..3), all of unit vectors
// and q with its scale.
struct __align__(16) GdnLengths { float ik, iq, kk[3], qk[4], pad[3]; };

namespace {

constexpr int kD = 128;        // head size of keys and values
constexpr int kCols = 32;      // value columns of a CTA
constexpr int kLanes = 16;     // lanes that share a column
constexpr int kThreads = kCols / 4 * kLanes;

// 8 lanes per (token, key head).
template <typename T, bool VEC>
__global__ void __launch_bounds__(256)
gdn_lengths_kernel(GdnLengths* out, const T* q, const T* k, int tokens, int hq,
                   int64_t q_stride, int64_t k_stride, float scale, int l2norm) {
  pdl_trigger();
  pdl_wait();
  const int64_t w = (int64_t)blockIdx.x * 32 + (threadIdx.x >> 3);
  const int lane = threadIdx.x & 7;
  const bool live = w < (int64_t)tokens * hq;
  const int t = live ? (int)(w / hq) : 0, h = live ? (int)(w % hq) : 0;
  uint4 raw[5][2];                        // q_t, k_t, k_{t-1} ..: all on their way at once (before the first token: the first)
#pragma unroll
  for (int r = 0; r < 5; ++r) {
    const T* at = (r == 0 ? q + t * q_stride : k + (int64_t)max(t - (r - 1), 0) * k_stride) + h * kD + lane * 8;
#pragma unroll
    for (int i = 0; i < 2; ++i) {         // entries lane * 8 and 64 + lane * 8 on
      if constexpr (VEC) {
        raw[r][i] = *reinterpret_cast<const uint4*>(at + i * 64);
      } else {
        T x[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = at[i * 64 + e];
        raw[r][i] = *reinterpret_cast<const uint4*>(x);
      }
    }
  }
  float s[8] = {}, kn[4] = {};            // |q|^2, q . k_{t-d}, k_t . k_{t-d}; |k_{t-d}|^2
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    float qv[8], kv[8];
    unpack8<T>(raw[0][i], qv);
    unpack8<T>(raw[1][i], kv);
#pragma unroll
    for (int e = 0; e < 8; ++e) s[0] = fmaf(qv[e], qv[e], s[0]);
#pragma unroll
    for (int d = 0; d < 4; ++d) {
      float x[8];
      unpack8<T>(raw[1 + d][i], x);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        kn[d] = fmaf(x[e], x[e], kn[d]);
        s[1 + d] = fmaf(qv[e], x[e], s[1 + d]);
        if (d > 0) s[4 + d] = fmaf(kv[e], x[e], s[4 + d]);
      }
    }
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) {
#pragma unroll
    for (int i = 0; i < 8; ++i) s[i] += __shfl_xor_sync(0xffffffffu, s[i], o);
#pragma unroll
    for (int i = 0; i < 4; ++i) kn[i] += __shfl_xor_sync(0xffffffffu, kn[i], o);
  }
  if (!live || lane != 0) return;
  GdnLengths r;
  float ik[4];
#pragma unroll
  for (int d = 0; d < 4; ++d) ik[d] = l2norm ? rsqrtf(kn[d] + 1e-6f) : 1.f;
  r.ik = ik[0];
  r.iq = (l2norm ? rsqrtf(s[0] + 1e-6f) : 1.f) * scale;
#pragma unroll
  for (int d = 0; d < 4; ++d) r.qk[d] = s[1 + d] * r.iq * ik[d];
#pragma unroll
  for (int d = 1; d < 4; ++d) r.kk[d - 1] = s[4 + d] * ik[0] * ik[d];
  r.pad[0] = r.pad[1] = r.pad[2] = 0.f;
  out[w] = r;
}

// log decay and beta of a token and head: given, or formed from the layer's projections as -exp(A) softplus(a + bias), sigmoid(b)
template <typename T>
__device__ __forceinline__ void gdn_gates(const GdnParams& p, int64_t t, int h, float& g, float& beta) {
  if (p.g != nullptr) {
    g = p.g[t * p.hv + h];
    beta = p.beta[t * p.hv + h];
    return;
  }
  const int rep = p.hv / p.hq;
  const T* row = reinterpret_cast<const T*>(p.ba) + t * p.ba_stride + (h / rep) * 2 * rep + h % rep;
  const float a = to_f(row[rep]) + p.dt_bias[h];
  const float sp = a > 20.f ? a : log1pf(expf(a));
  g = -expf(p.a_log[h]) * sp;
  beta = 1.f / (1.f + expf(-to_f(row[0])));
}

// VEC: rows can be read 16 bytes at a time.
template <typename T, bool VEC>
__global__ void __launch_bounds__(kThreads, 3)
gdn_kernel(const GdnParams p) {
  pdl_trigger();
  pdl_wait();
  constexpr int G = 4, NS = 16, NB = 2;                        // tokens of a group, of a stage; stages
  constexpr int KQ = NS * (kD / 8) / kThreads;
  const int b = blockIdx.z, h = blockIdx.y, hk = h / (p.hv / p.hq), col0 = blockIdx.x * kCols;
  const int64_t t0 = p.query_start_loc[b], t1 = p.query_start_loc[b + 1];
  if ((int)t1 - (int)t0 <= p.short_len) return;
  __shared__ __align__(16) float s_k[NB][NS][kD], s_q[NB][NS][kD];
  __shared__ __align__(16) T s_v[NB][NS][kCols], s_o[NB][NS][kCols];
  __shared__ __align__(16) float s_c[NB][NS][12];              // beta|k|^-1 e^G, beta, q e^G, update's factor; L x 3, e^G_last; M x 4
  __shared__ __align__(16) float s_w[kThreads / kLanes][G][4];
  const int tid = threadIdx.x, rl = tid % kLanes, cg = tid / kLanes, c4 = cg * 4;
  const int slot = p.state_idx ? p.state_idx[b] : -1;
  float* st = slot >= 0 ? p.state + (((int64_t)slot * p.hv + h) * kD) * kD + col0 + c4 : nullptr;
  const T *gq = reinterpret_cast<const T*>(p.q) + hk * kD, *gk = reinterpret_cast<const T*>(p.k) + hk * kD,
          *gv = reinterpret_cast<const T*>(p.v) + h * kD + col0;
  T* go = reinterpret_cast<T*>(p.out) + (int64_t)h * kD + col0;

  auto read8 = [&](const T* at, bool live) {
    uint4 r = make_uint4(0u, 0u, 0u, 0u);
    if (!live) return r;
    if constexpr (VEC) {
      r = *reinterpret_cast<const uint4*>(at);
    } else {
      T x[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) x[e] = at[e];
      r = *reinterpret_cast<const uint4*>(x);
    }
    return r;
  };
  uint4 nk[KQ], nq[KQ], nv;
  auto fetch = [&](int64_t tc) {
#pragma unroll
    for (int i = 0; i < KQ; ++i) {
      const int at = tid + i * kThreads, r = at / (kD / 8), c = at % (kD / 8) * 8;
      const bool live = r < NS && tc + r < t1;
      nk[i] = read8(gk + (tc + r) * p.k_stride + c, live);
      nq[i] = read8(gq + (tc + r) * p.q_stride + c, live);
    }
    const int r = tid / (kCols / 8), c = tid % (kCols / 8) * 8;
    nv = read8(gv + (tc + r) * p.v_stride + c, r < NS && tc + r < t1);
  };
  // what the fetch brought, and the factors of a stage's tokens (a thread each)
  auto store = [&](int64_t tc, int buf) {
#pragma unroll
    for (int i = 0; i < KQ; ++i) {
      const int at = tid + i * kThreads, r = at / (kD / 8), c = at % (kD / 8) * 8;
      if (r >= NS) break;
      float x[8];
      unpack8<T>(nk[i], x);
      *reinterpret_cast<float4*>(&s_k[buf][r][c]) = make_float4(x[0], x[1], x[2], x[3]);
      *reinterpret_cast<float4*>(&s_k[buf][r][c + 4]) = make_float4(x[4], x[5], x[6], x[7]);
      unpack8<T>(nq[i], x);
      *reinterpret_cast<float4*>(&s_q[buf][r][c]) = make_float4(x[0], x[1], x[2], x[3]);
      *reinterpret_cast<float4*>(&s_q[buf][r][c + 4]) = make_float4(x[4], x[5], x[6], x[7]);
    }
    if (tid / (kCols / 8) < NS) *reinterpret_cast<uint4*>(&s_v[buf][tid / (kCols / 8)][tid % (kCols / 8) * 8]) = nv;
    {
      if (tid < 32) {                                          // (a whole warp: gates are exchanged; tokens in the first half)
        const int64_t t = tc + tid;
        const bool live = tid < NS && t < t1;
        float g = 0.f, beta = 0.f;
        GdnLengths len = {};
        if (live) {
          gdn_gates<T>(p, t, h, g, beta);
          len = p.lengths[t * p.hq + hk];
        }
        const int j = tid % G;
        float sum[G];                                          // g of this token, of it and the one before, ..
        sum[0] = g;
#pragma unroll
        for (int d = 1; d < G; ++d) sum[d] = sum[d - 1] + __shfl_up_sync(0xffffffffu, g, d);
        float upto = sum[0], after = 0.f;                      // from the group's first token on; behind this token
#pragma unroll
        for (int d = 1; d < G; ++d) {
          if (d <= j) upto = sum[d];
          const float x = __shfl_down_sync(0xffffffffu, g, d);
          if (j + d < G) after += x;
        }
        if (tid < NS) {
          float* c = s_c[buf][tid];
          const float e = expf(upto);
          c[0] = beta * len.ik * e;
          c[1] = beta;
          c[2] = len.iq * e;
          c[3] = expf(after) * len.ik;
#pragma unroll
          for (int d = 1; d < G; ++d) c[3 + d] = d <= j ? beta * expf(sum[d - 1]) * len.kk[d - 1] : 0.f;
          c[7] = e;
          c[8] = len.qk[0];
#pragma unroll
          for (int d = 1; d < G; ++d) c[8 + d] = d <= j ? expf(sum[d - 1]) * len.qk[d] : 0.f;
        }
      }
    }
  };
  auto flush = [&](int64_t tc, int buf) {
    const int r = tid / (kCols / 8), c = tid % (kCols / 8) * 8;
    if (r < NS && tc + r < t1)
      *reinterpret_cast<uint4*>(go + (tc + r) * p.hv * kD + c) = *reinterpret_cast<const uint4*>(&s_o[buf][r][c]);
  };

  fetch(t0);
  uint64_t S[4][4];                                            // rows (2i, 2i + 1) of the lane's eight, four columns
  {
    const bool init = st != nullptr && (p.has_initial == nullptr || p.has_initial[b] != 0);
    float4 x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int row = (i / 4) * 64 + rl * 4 + i % 4;
      x[i] = init ? *reinterpret_cast<const float4*>(st + (int64_t)row * kD) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      S[i][0] = pack2f(x[2 * i].x, x[2 * i + 1].x);
      S[i][1] = pack2f(x[2 * i].y, x[2 * i + 1].y);
      S[i][2] = pack2f(x[2 * i].z, x[2 * i + 1].z);
      S[i][3] = pack2f(x[2 * i].w, x[2 * i + 1].w);
    }
  }
  store(t0, 0);
  __syncthreads();
  int buf = 0;
  for (int64_t tc = t0; tc < t1; tc += NS) {
    const bool more = tc + NS < t1;
    if (more) fetch(tc + NS);
    if (tc > t0) flush(tc - NS, buf ^ 1);
    const int n = (int)min((int64_t)NS, t1 - tc);
    for (int s = 0; s < n; s += G) {
      uint64_t acc[2 * G][4];                                  // k_t . S, then q_t . S
#pragma unroll
      for (int half = 0; half < 2; ++half)
#pragma unroll
        for (int t = 0; t < 2 * G; ++t) {
          const float* row = (t < G ? s_k[buf][s + t] : s_q[buf][s + t - G]) + half * 64 + rl * 4;
          const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(row);
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            acc[t][c] = half == 0 ? mul2f(x.x, S[0][c]) : fma2f(x.x, S[2][c], acc[t][c]);
            acc[t][c] = fma2f(x.y, S[2 * half + 1][c], acc[t][c]);
          }
        }
      // one column and, of its sums, those with k or those with q per pair of lanes
      const int lc = (rl >> 2) & 3;                            // column
      const bool isq = (rl >> 1) & 1;
      float d[G];
      {
        float a[2 * G][4];
#pragma unroll
        for (int t = 0; t < 2 * G; ++t)
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            float lo, hi;
            unpack2f(acc[t][c], lo, hi);
            a[t][c] = lo + hi;
          }
        const bool h3 = rl & 8, h2 = rl & 4;
        float a2[2 * G][2];
#pragma unroll
        for (int t = 0; t < 2 * G; ++t)
#pragma unroll
          for (int c = 0; c < 2; ++c)
            a2[t][c] = (h3 ? a[t][2 + c] : a[t][c]) + __shfl_xor_sync(0xffffffffu, h3 ? a[t][c] : a[t][2 + c], 8);
        float a1[2 * G];
#pragma unroll
        for (int t = 0; t < 2 * G; ++t)
          a1[t] = (h2 ? a2[t][1] : a2[t][0]) + __shfl_xor_sync(0xffffffffu, h2 ? a2[t][0] : a2[t][1], 4);
#pragma unroll
        for (int t = 0; t < G; ++t) {
          d[t] = (isq ? a1[G + t] : a1[t]) + __shfl_xor_sync(0xffffffffu, isq ? a1[t] : a1[G + t], 2);
          d[t] += __shfl_xor_sync(0xffffffffu, d[t], 1);
        }
      }
      float u[G], last;
      {
        float cf[G][12];
#pragma unroll
        for (int t = 0; t < G; ++t)
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            const float4 x = *reinterpret_cast<const float4*>(&s_c[buf][s + t][4 * i]);
            cf[t][4 * i] = x.x; cf[t][4 * i + 1] = x.y; cf[t][4 * i + 2] = x.z; cf[t][4 * i + 3] = x.w;
          }
        last = cf[G - 1][7];
#pragma unroll
        for (int t = 0; t < G; ++t) {                          // (lanes with q sums compute along and drop it)
          u[t] = fmaf(cf[t][1], to_f(s_v[buf][s + t][c4 + lc]), -cf[t][0] * d[t]);
#pragma unroll
          for (int j = 0; j < t; ++j) u[t] = fmaf(-cf[t][3 + t - j], u[j], u[t]);
        }
        float uk[G];
#pragma unroll
        for (int t = 0; t < G; ++t) uk[t] = __shfl_xor_sync(0xffffffffu, u[t], 2);
        if (isq) {
#pragma unroll
          for (int t = 0; t < G; ++t) {
            float o = cf[t][2] * d[t];
#pragma unroll
            for (int j = 0; j <= t; ++j) o = fmaf(cf[t][8 + t - j], uk[j], o);
            if ((t & 1) == (rl & 1)) s_o[buf][s + t][c4 + lc] = from_f<T>(o);
          }
        } else {
#pragma unroll
          for (int t = 0; t < G; ++t)
            if ((t & 1) == (rl & 1)) s_w[cg][t][lc] = cf[t][3] * u[t];
        }
      }
      __syncwarp();
      const uint64_t dl = pack2f(last, last);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) S[i][c] = mul2f(S[i][c], dl);
#pragma unroll
      for (int t = 0; t < G; ++t) {
        const float4 w = *reinterpret_cast<const float4*>(s_w[cg][t]);
        const uint64_t wc[4] = {pack2f(w.x, w.x), pack2f(w.y, w.y), pack2f(w.z, w.z), pack2f(w.w, w.w)};
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(s_k[buf][s + t] + half * 64 + rl * 4);
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            S[2 * half][c] = fma2f(x.x, wc[c], S[2 * half][c]);
            S[2 * half + 1][c] = fma2f(x.y, wc[c], S[2 * half + 1][c]);
          }
        }
      }
      __syncwarp();                                            // s_w is rewritten by the next group
    }
    if (more) store(tc + NS, buf ^ 1);
    __syncthreads();
    if (!more) flush(tc, buf);
    buf ^= 1;
  }
  if (st != nullptr) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float x[2][4];
#pragma unroll
      for (int c = 0; c < 4; ++c) unpack2f(S[i][c], x[0][c], x[1][c]);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int row = (i / 2) * 64 + rl * 4 + (i % 2) * 2 + e;
        *reinterpret_cast<float4*>(st + (int64_t)row * kD) = make_float4(x[e][0], x[e][1], x[e][2], x[e][3]);
      }
    }
  }
}

// ------------------------------------------------------------------------------------------ chunks of 16 tokens (bf16)
// The recurrence over a chunk as products of 16 x 16 and 16 x 128 matrices on the tensor cores: with L_tj = beta_t D_tj k_t . k_j
// (j < t), U = (I + L)^-1 (beta V - A K S), O = C Q S + M U, S <- e^G S + K^T (W U), where A, C and W are factors per token.  What
// depends on q, k and the gates alone comes from a kernel in front, for all chunks at once.  q and k are the 16-bit rows
// themselves; everything of 32 bits (the state, U) goes in as three bf16 terms, which hold its 24 bits, so the products are as
// exact as fp32 ones.  Bound by the mma.sync rate along the longest sequence: 144 products a chunk and warp.
constexpr int kC = 16;                     // tokens of a chunk
constexpr int kChunkFloats = 2 * kC * kC + 5 * kC;   // T, M; factors a, beta, c, w; e^G of the last token

__device__ __forceinline__ int gdn_chunks(const GdnParams& p, int b) {
  const int n = p.query_start_loc[b + 1] - p.query_start_loc[b];
  return n > p.short_len ? (n + kC - 1) / kC : 0;
}

// The chunk of index `at` in the order of the sequences: its sequence and first token, or false behind the last.  A whole warp.
__device__ __forceinline__ bool gdn_locate(const GdnParams& p, int at, int lane, int& seq, int& first, int& end) {
  int before = 0;
  for (int b0 = 0; b0 < p.batch; b0 += 32) {
    const int b = b0 + lane;
    const int n = b < p.batch ? gdn_chunks(p, b) : 0;
    int inc = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += v;
    }
    const unsigned hit = __ballot_sync(0xffffffffu, at < before + inc);
    if (hit) {
      const int src = __ffs(hit) - 1;
      const int start = before + __shfl_sync(0xffffffffu, inc - n, src);
      seq = b0 + src;
      first = p.query_start_loc[seq] + (at - start) * kC;
      end = p.query_start_loc[seq + 1];
      return true;
    }
    before += __shfl_sync(0xffffffffu, inc, 31);
  }
  return false;
}

// Rows t0 .. of n tokens, kD entries each, as bf16 with swizzled 16-byte chunks; rows from n on are zero.
template <bool VEC>
__device__ __forceinline__ void gdn_copy_rows(__nv_bfloat16* dst, const __nv_bfloat16* src, int64_t stride, int n, int tid,
                                              int threads) {
  for (int i = tid; i < kC * (kD / 8); i += threads) {
    const int r = i / (kD / 8), c = i % (kD / 8);
    void* d = dst + r * kD + ((c ^ (r & 7)) * 8);
    const __nv_bfloat16* at = src + r * stride + c * 8;
    if constexpr (VEC) {
      cp_async16(d, r < n ? at : src, r < n);
    } else {
      __nv_bfloat16 x[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) x[e] = r < n ? at[e] : __float2bfloat16_rn(0.f);
      *reinterpret_cast<uint4*>(d) = *reinterpret_cast<const uint4*>(x);
    }
  }
}

// One CTA per (chunk, key head), a warp per value head of it in turn: (I + L)^-1 with L_tj = beta_t D_tj k_t . k_j (j < t), M_tj =
// D_tj q_t . k_j (j <= t), both of unit vectors, and the factors of the sums with the state.
template <bool VEC>
__global__ void __launch_bounds__(128)
gdn_chunk_prepare_kernel(const GdnParams p) {
  using T = __nv_bfloat16;
  pdl_trigger();
  pdl_wait();
  __shared__ __align__(128) T s_k[kC * kD], s_q[kC * kD];
  __shared__ float s_kk[kC][kC], s_qk[kC][kC], s_ik[kC], s_iq[kC], s_l[4][kC][kC + 1];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, hk = blockIdx.y;
  int seq, first, end;
  if (!gdn_locate(p, blockIdx.x, lane, seq, first, end)) return;
  const int n = min(kC, end - first);
  gdn_copy_rows<VEC>(s_k, reinterpret_cast<const T*>(p.k) + first * p.k_stride + hk * kD, p.k_stride, n, tid, 128);
  gdn_copy_rows<VEC>(s_q, reinterpret_cast<const T*>(p.q) + first * p.q_stride + hk * kD, p.q_stride, n, tid, 128);
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  if (warp < 2) {                                   // k k^T, q k^T: the products of bf16 are exact, their sums in fp32
    float d[2][4] = {};
    const T* a = warp == 0 ? s_k : s_q;
#pragma unroll
    for (int ks = 0; ks < kD / 16; ++ks) {
      uint32_t af[4], bf[4];
      const int mat = lane >> 3;
      const int ra = (mat & 1) * 8 + (lane & 7), rb = (mat >> 1) * 8 + (lane & 7);
      ldmatrix_x4(af, a + ra * kD + (((2 * ks + (mat >> 1)) ^ (ra & 7)) * 8));
      ldmatrix_x4(bf, s_k + rb * kD + (((2 * ks + (mat & 1)) ^ (rb & 7)) * 8));
      mma16816<T>(d[0], af, bf[0], bf[1]);
      mma16816<T>(d[1], af, bf[2], bf[3]);
    }
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        (warp == 0 ? s_kk : s_qk)[(lane >> 2) + (e >> 1) * 8][nt * 8 + 2 * (lane & 3) + (e & 1)] = d[nt][e];
  } else if (warp == 2) {                           // |q|^2, two lanes a token
    const int r = lane >> 1;
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float f[8];
      unpack8<T>(*reinterpret_cast<const uint4*>(s_q + r * kD + ((((lane & 1) * 8 + i) ^ (r & 7)) * 8)), f);
#pragma unroll
      for (int e = 0; e < 8; ++e) ss = fmaf(f[e], f[e], ss);
    }
    ss += __shfl_xor_sync(0xffffffffu, ss, 1);
    if (!(lane & 1)) s_iq[r] = (p.l2norm ? rsqrtf(ss + 1e-6f) : 1.f) * p.scale;
  }
  __syncthreads();
  if (tid < kC) s_ik[tid] = p.l2norm ? rsqrtf(s_kk[tid][tid] + 1e-6f) : 1.f;
  __syncthreads();
  const int rep = p.hv / p.hq;
  for (int hr = warp; hr < rep; hr += 4) {
    const int h = hk * rep + hr, t = lane & (kC - 1);
    float g = 0.f, beta = 0.f;
    if (t < n) gdn_gates<T>(p, first + t, h, g, beta);
    float upto = g;                                 // sums over the chunk's tokens up to this one
#pragma unroll
    for (int o = 1; o < kC; o <<= 1) {
      const float v = __shfl_up_sync(0xffffffffu, upto, o, kC);
      if (t >= o) upto += v;
    }
    const float all = __shfl_sync(0xffffffffu, upto, kC - 1, kC);
    float* out = const_cast<float*>(p.chunks) + ((int64_t)blockIdx.x * p.hv + h) * kChunkFloats;
    float after = 0.f;                              // those behind this token, summed by themselves
    {
      float v = __shfl_down_sync(0xffffffffu, g, 1, kC);
      after = t + 1 < kC ? v : 0.f;
#pragma unroll
      for (int o = 1; o < kC; o <<= 1) {
        v = __shfl_down_sync(0xffffffffu, after, o, kC);
        if (t + o < kC) after += v;
      }
    }
    if (lane < kC) {
      const float e = expf(upto), ik = s_ik[t];
      float* f = out + 2 * kC * kC;
      f[t] = beta * e * ik;
      f[kC + t] = beta;
      f[2 * kC + t] = s_iq[t] * e;
      f[3 * kC + t] = expf(after) * ik;
      if (t == 0) f[4 * kC] = expf(all);
    }
    // lanes t and t + 16: every other column j.  D_tj = exp(g_{j+1} + .. + g_t), each sum by itself
    float between = 0.f;
#pragma unroll
    for (int j = kC - 1; j >= 0; --j) {
      const float gj = __shfl_sync(0xffffffffu, g, (j + 1) & (kC - 1), kC);
      if (j < t) between += gj;
      if ((j & 1) != (lane >> 4)) continue;
      const float d = expf(between);
      s_l[warp][t][j] = j < t ? beta * d * s_kk[t][j] * s_ik[t] * s_ik[j] : 0.f;
      out[kC * kC + t * kC + j] = j <= t ? d * s_qk[t][j] * s_iq[t] * s_ik[j] : 0.f;
    }
    __syncwarp();
    if (lane < kC) {                                // column `lane` of the inverse by forward substitution
      float x[kC];
#pragma unroll
      for (int r = 0; r < kC; ++r) {
        float v = r == lane ? 1.f : 0.f;
#pragma unroll
        for (int j = 0; j < r; ++j) v = fmaf(-s_l[warp][r][j], x[j], v);
        x[r] = v;
        out[r * kC + lane] = v;
      }
    }
    __syncwarp();
  }
}

// fp32 pairs as three bf16 terms each, which hold all 24 bits.
__device__ __forceinline__ void split3(float a, float b, uint32_t (&t)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    t[i] = *reinterpret_cast<const uint32_t*>(&v);
    a -= __uint_as_float(t[i] << 16);
    b -= __uint_as_float(t[i] & 0xffff0000u);
  }
}

constexpr int kWarpCols = 16, kChunkWarps = 4, kPadR = kC + 2;

// One CTA = one (sequence, value head, 64 value columns), a warp 16 columns of the state, transposed, as accumulators of
// m16n8k16: they are the second operand of the products with k and q as they stand, and take the update as products with k.
template <bool VEC>
__global__ void __launch_bounds__(kChunkWarps * 32, 2)
gdn_chunk_kernel(const GdnParams p) {
  using T = __nv_bfloat16;
  constexpr int CV = kWarpCols * kChunkWarps, TH = kChunkWarps * 32;
  pdl_trigger();
  pdl_wait();
  __shared__ __align__(128) T s_k[2][kC * kD], s_q[2][kC * kD];
  __shared__ __align__(16) T s_v[2][kC][CV];
  __shared__ __align__(16) float s_f[2][kChunkFloats];
  __shared__ __align__(16) float s_r[kChunkWarps][kC][kPadR], s_d[kChunkWarps][kC][kPadR];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gq = lane >> 2, tl = lane & 3;
  const int b = blockIdx.z, h = blockIdx.y, hk = h / (p.hv / p.hq), col0 = blockIdx.x * CV + warp * kWarpCols;
  const int t0 = p.query_start_loc[b], t1 = p.query_start_loc[b + 1];
  if (t1 <= t0 + p.short_len) return;
  int chunk = 0;                                    // index of the sequence's first chunk
  for (int i = lane; i < b; i += 32) chunk += gdn_chunks(p, i);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) chunk += __shfl_xor_sync(0xffffffffu, chunk, o);
  const int slot = p.state_idx ? p.state_idx[b] : -1;
  float* st = slot >= 0 ? p.state + (((int64_t)slot * p.hv + h) * kD) * kD + col0 : nullptr;
  const T *gk = reinterpret_cast<const T*>(p.k) + hk * kD, *gqr = reinterpret_cast<const T*>(p.q) + hk * kD,
          *gv = reinterpret_cast<const T*>(p.v) + h * kD + blockIdx.x * CV;
  auto fetch = [&](int tc, int at, int buf) {
    const int n = min(kC, t1 - tc);
    gdn_copy_rows<VEC>(s_k[buf], gk + tc * p.k_stride, p.k_stride, n, tid, TH);
    gdn_copy_rows<VEC>(s_q[buf], gqr + tc * p.q_stride, p.q_stride, n, tid, TH);
    {
      const int r = tid / (CV / 8), c = tid % (CV / 8) * 8;            // (128 threads: 16 rows of 8 pieces)
      const T* at8 = gv + (int64_t)(tc + r) * p.v_stride + c;
      if constexpr (VEC) {
        cp_async16(&s_v[buf][r][c], r < n ? at8 : gv, r < n);
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) s_v[buf][r][c + e] = r < n ? at8[e] : __float2bfloat16_rn(0.f);
      }
    }
    const float* f = p.chunks + ((int64_t)at * p.hv + h) * kChunkFloats;
    for (int i = tid; i < kChunkFloats / 4; i += TH) cp_async16(&s_f[buf][i * 4], f + i * 4, true);
    cp_async_commit();
  };
  static_assert(TH == kC * (CV / 8) && kChunkFloats % 4 == 0, "one piece of v a thread");
  fetch(t0, chunk, 0);
  float S[kD / 8][4];                               // keys 8 i + 2 tl, + 1 of columns gq and gq + 8
  {
    const bool init = st != nullptr && (p.has_initial == nullptr || p.has_initial[b] != 0);
#pragma unroll
    for (int i = 0; i < kD / 8; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) S[i][e] = init ? st[(int64_t)(8 * i + 2 * tl + (e & 1)) * kD + gq + (e >> 1) * 8] : 0.f;
  }
  int buf = 0;
  for (int tc = t0; tc < t1; tc += kC, ++chunk, buf ^= 1) {
    cp_async_wait<0>();
    __syncthreads();                                // this chunk is here; the other buffer has been used up
    if (tc + kC < t1) fetch(tc + kC, chunk + 1, buf ^ 1);
    const float *fT = s_f[buf], *fM = fT + kC * kC, *fa = fM + kC * kC, *fb = fa + kC, *fc = fb + kC, *fw = fc + kC;
    // ---- k . S and q . S: [16 tokens] x [columns 0..7, 8..15 of the warp]
    float dk[2][4] = {}, dq[2][4] = {};
#pragma unroll
    for (int ks = 0; ks < kD / 16; ++ks) {
      uint32_t ka[4], qa[4];
      const int mat = lane >> 3, r = (mat & 1) * 8 + (lane & 7), o = r * kD + (((2 * ks + (mat >> 1)) ^ (r & 7)) * 8);
      ldmatrix_x4(ka, s_k[buf] + o);
      ldmatrix_x4(qa, s_q[buf] + o);
#pragma unroll
      for (int cg = 0; cg < 2; ++cg) {
        uint32_t lo[3], hi[3];
        split3(S[2 * ks][2 * cg], S[2 * ks][2 * cg + 1], lo);
        split3(S[2 * ks + 1][2 * cg], S[2 * ks + 1][2 * cg + 1], hi);
#pragma unroll
        for (int i = 2; i >= 0; --i) {
          mma16816<T>(dk[cg], ka, lo[i], hi[i]);
          mma16816<T>(dq[cg], qa, lo[i], hi[i]);
        }
      }
    }
    // ---- right-hand sides, then a column per pair of lanes
#pragma unroll
    for (int cg = 0; cg < 2; ++cg)
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        const int t = gq + hf * 8, c = cg * 8 + 2 * tl;
        const __nv_bfloat162 v = *reinterpret_cast<const __nv_bfloat162*>(&s_v[buf][t][warp * kWarpCols + c]);
        *reinterpret_cast<float2*>(&s_r[warp][t][c]) = make_float2(fb[t] * __low2float(v) - fa[t] * dk[cg][2 * hf],
                                                                   fb[t] * __high2float(v) - fa[t] * dk[cg][2 * hf + 1]);
        *reinterpret_cast<float2*>(&s_d[warp][t][c]) = make_float2(dq[cg][2 * hf], dq[cg][2 * hf + 1]);
      }
    __syncwarp();
    const int col = lane & 15, half = lane >> 4;    // this lane: rows 2 i + half
    float R[kC], u[8], U[kC];
#pragma unroll
    for (int t = 0; t < kC; ++t) R[t] = s_r[warp][t][col];
    // Row 2 i + half of a lower triangle times x.  Entries behind the row's own token are left out: the triangle's zeros would make
    // a NaN of an infinity or NaN there.
    auto rows = [&](const float* m, const float (&x)[kC], int i) {
      float acc = 0.f;
#pragma unroll
      for (int j = 0; j <= 2 * i; j += 4) {
        const float4 a = *reinterpret_cast<const float4*>(m + (2 * i + half) * kC + j);
        const float f[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (j + e <= 2 * i + 1) acc = fmaf(f[e], j + e <= 2 * i || half ? x[j + e] : 0.f, acc);
      }
      return acc;
    };
#pragma unroll
    for (int i = 0; i < 8; ++i) u[i] = rows(fT, R, i);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float other = __shfl_xor_sync(0xffffffffu, u[i], 16);
      U[2 * i] = half ? other : u[i];
      U[2 * i + 1] = half ? u[i] : other;
    }
    __syncwarp();                                   // (s_r has been read: it takes the update, columns first)
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int t = 2 * i + half;
      const float o = fmaf(fc[t], s_d[warp][t][col], rows(fM, U, i));
      if (tc + t < t1) reinterpret_cast<T*>(p.out)[((int64_t)(tc + t) * p.hv + h) * kD + col0 + col] = __float2bfloat16_rn(o);
      s_r[warp][col][t] = fw[t] * u[i];
    }
    __syncwarp();
    // ---- S <- e^G S + W^T k
    uint32_t w[4][3];
    {
      float2 x = *reinterpret_cast<const float2*>(&s_r[warp][gq][2 * tl]);
      split3(x.x, x.y, w[0]);
      x = *reinterpret_cast<const float2*>(&s_r[warp][gq + 8][2 * tl]);
      split3(x.x, x.y, w[1]);
      x = *reinterpret_cast<const float2*>(&s_r[warp][gq][2 * tl + 8]);
      split3(x.x, x.y, w[2]);
      x = *reinterpret_cast<const float2*>(&s_r[warp][gq + 8][2 * tl + 8]);
      split3(x.x, x.y, w[3]);
    }
    const float last = fw[kC];
#pragma unroll
    for (int i = 0; i < kD / 8; i += 2) {
      uint32_t kt[4];
      const int mat = lane >> 3, r = (mat & 1) * 8 + (lane & 7);
      ldmatrix_x4_trans(kt, s_k[buf] + r * kD + (((i + (mat >> 1)) ^ (r & 7)) * 8));
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        S[i][e] *= last;
        S[i + 1][e] *= last;
      }
#pragma unroll
      for (int j = 2; j >= 0; --j) {
        const uint32_t a[4] = {w[0][j], w[1][j], w[2][j], w[3][j]};
        mma16816<T>(S[i], a, kt[0], kt[1]);
        mma16816<T>(S[i + 1], a, kt[2], kt[3]);
      }
    }
    __syncwarp();                                   // s_r, s_d are rewritten by the next chunk
  }
  if (st != nullptr) {
#pragma unroll
    for (int i = 0; i < kD / 8; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) st[(int64_t)(8 * i + 2 * tl + (e & 1)) * kD + gq + (e >> 1) * 8] = S[i][e];
  }
}

// Short sequences: one CTA = one (sequence, value head), tokens one at a time.  A warp holds 16 rows of S, a lane 4 columns of them, so
// that a warp reads and writes whole rows of 512 bytes, all before the first product; the warps' sums meet in shared memory.
template <typename T>
__global__ void __launch_bounds__(256, 2)
gdn_step_kernel(const GdnParams p) {
  pdl_trigger();
  pdl_wait();
  const int b = blockIdx.x, h = blockIdx.y, hk = h / (p.hv / p.hq), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t t0 = p.query_start_loc[b], t1 = p.query_start_loc[b + 1];
  if (t1 <= t0 || (!p.step && t1 - t0 > p.short_len)) return;
  __shared__ __align__(16) float s_sum[2][2][8][kD];           // (two sets: a token is one barrier)
  const int slot = p.state_idx ? p.state_idx[b] : -1;
  const bool init = slot >= 0 && (p.has_initial == nullptr || p.has_initial[b] != 0);
  float* st = slot >= 0 ? p.state + (((int64_t)slot * p.hv + h) * kD + warp * 16) * kD + lane * 4 : nullptr;
  float4 S[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) S[i] = init ? *reinterpret_cast<const float4*>(st + i * kD) : make_float4(0.f, 0.f, 0.f, 0.f);
  int buf = 0;
  for (int64_t t = t0; t < t1; ++t, buf ^= 1) {
    const T *q = reinterpret_cast<const T*>(p.q) + t * p.q_stride + hk * kD, *k = reinterpret_cast<const T*>(p.k) + t * p.k_stride + hk * kD,
            *v = reinterpret_cast<const T*>(p.v) + t * p.v_stride + h * kD;
    float qv[4], kv[4], qq = 0.f, kk = 0.f, qk = 0.f, g, beta;
    gdn_gates<T>(p, t, h, g, beta);
#pragma unroll
    for (int i = 0; i < 4; ++i) {                              // every warp has the rows whole, for their lengths
      qv[i] = to_f(q[lane * 4 + i]);
      kv[i] = to_f(k[lane * 4 + i]);
      qq = fmaf(qv[i], qv[i], qq);
      kk = fmaf(kv[i], kv[i], kk);
      qk = fmaf(qv[i], kv[i], qk);
    }
    qq = warp_sum(qq); kk = warp_sum(kk); qk = warp_sum(qk);
    const float ik = p.l2norm ? rsqrtf(kk + 1e-6f) : 1.f, iq = (p.l2norm ? rsqrtf(qq + 1e-6f) : 1.f) * p.scale, decay = expf(g);
    float kr[16], ks[4] = {}, qs[4] = {};                      // a warp's rows of k from its lanes
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const int src = warp * 4 + i / 4;
      kr[i] = __shfl_sync(0xffffffffu, kv[i % 4], src) * ik;
      const float qr = __shfl_sync(0xffffffffu, qv[i % 4], src) * iq;
      ks[0] = fmaf(S[i].x, kr[i], ks[0]); ks[1] = fmaf(S[i].y, kr[i], ks[1]);
      ks[2] = fmaf(S[i].z, kr[i], ks[2]); ks[3] = fmaf(S[i].w, kr[i], ks[3]);
      qs[0] = fmaf(S[i].x, qr, qs[0]); qs[1] = fmaf(S[i].y, qr, qs[1]);
      qs[2] = fmaf(S[i].z, qr, qs[2]); qs[3] = fmaf(S[i].w, qr, qs[3]);
    }
    *reinterpret_cast<float4*>(&s_sum[buf][0][warp][lane * 4]) = make_float4(ks[0], ks[1], ks[2], ks[3]);
    *reinterpret_cast<float4*>(&s_sum[buf][1][warp][lane * 4]) = make_float4(qs[0], qs[1], qs[2], qs[3]);
    __syncthreads();
    float u[4] = {}, o[4] = {};
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      const float4 x = *reinterpret_cast<const float4*>(&s_sum[buf][0][w][lane * 4]);
      u[0] += x.x; u[1] += x.y; u[2] += x.z; u[3] += x.w;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) u[i] = beta * (to_f(v[lane * 4 + i]) - decay * u[i]);
    if (warp == 0) {
#pragma unroll
      for (int w = 0; w < 8; ++w) {
        const float4 x = *reinterpret_cast<const float4*>(&s_sum[buf][1][w][lane * 4]);
        o[0] += x.x; o[1] += x.y; o[2] += x.z; o[3] += x.w;
      }
      T* out = reinterpret_cast<T*>(p.out) + (t * p.hv + h) * kD + lane * 4;
#pragma unroll
      for (int i = 0; i < 4; ++i) out[i] = from_f<T>(decay * o[i] + qk * ik * iq * u[i]);
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      S[i].x = fmaf(kr[i], u[0], decay * S[i].x); S[i].y = fmaf(kr[i], u[1], decay * S[i].y);
      S[i].z = fmaf(kr[i], u[2], decay * S[i].z); S[i].w = fmaf(kr[i], u[3], decay * S[i].w);
    }
  }
  if (st != nullptr) {
#pragma unroll
    for (int i = 0; i < 16; ++i) *reinterpret_cast<float4*>(st + i * kD) = S[i];
  }
}

int64_t gdn_max_chunks(int64_t tokens, int batch) { return tokens / kC + batch; }

template <typename T>
void launch(const GdnParams& p, cudaStream_t stream) {
  auto wide = [](const void* at, int64_t stride) { return (reinterpret_cast<uintptr_t>(at) & 15) == 0 && stride % 8 == 0; };
  const bool vec = wide(p.q, p.q_stride) && wide(p.k, p.k_stride) && wide(p.v, p.v_stride);
  const dim3 grid(kD / kCols, p.hv, p.batch);
  if (p.step || p.short_len > 0) pdl_run(gdn_step_kernel<T>, dim3(p.batch, p.hv), 256, 0, stream, p);
  if (p.step) return;
  if constexpr (std::is_same<T, __nv_bfloat16>::value) {
    const dim3 chunks((unsigned)gdn_max_chunks(p.tokens, p.batch), p.hq), parts(kD / (kWarpCols * kChunkWarps), p.hv, p.batch);
    if (vec) {
      pdl_run(gdn_chunk_prepare_kernel<true>, chunks, 128, 0, stream, p);
      pdl_run(gdn_chunk_kernel<true>, parts, kChunkWarps * 32, 0, stream, p);
    } else {
      pdl_run(gdn_chunk_prepare_kernel<false>, chunks, 128, 0, stream, p);
      pdl_run(gdn_chunk_kernel<false>, parts, kChunkWarps * 32, 0, stream, p);
    }
  } else {
    const unsigned blocks = (unsigned)((p.tokens * p.hq + 31) / 32);
    GdnLengths* len = const_cast<GdnLengths*>(p.lengths);
#define GDN_RUN(V)                                                                                                            \
  pdl_run(gdn_lengths_kernel<T, V>, blocks, 256, 0, stream, len, (const T*)p.q, (const T*)p.k, (int)p.tokens, p.hq, p.q_stride, \
          p.k_stride, p.scale, p.l2norm);                                                                                     \
  pdl_run(gdn_kernel<T, V>, grid, kThreads, 0, stream, p)
    if (vec) { GDN_RUN(true); } else { GDN_RUN(false); }
#undef GDN_RUN
  }
}

// DIM / 8 lanes per (token, head).
template <typename T, int DIM>
__global__ void __launch_bounds__(256)
gated_head_norm_kernel(T* out, const T* o, const T* z, const T* w,
                       int64_t rows, int heads, int rep, int64_t z_stride, int64_t z_group, float eps) {
  pdl_trigger();
  pdl_wait();
  constexpr int L = DIM / 8;
  const int64_t r = (int64_t)blockIdx.x * (256 / L) + threadIdx.x / L;
  const int c = threadIdx.x % L * 8;
  const bool live = r < rows;
  const int64_t t = live ? r / heads : 0;
  const int h = live ? (int)(r % heads) : 0;
  const T* zr = z + t * z_stride + (h / rep) * z_group + (h % rep) * DIM + c;
  float f[8] = {}, g[8] = {};
  if (live) {
    unpack8<T>(*reinterpret_cast<const uint4*>(o + r * DIM + c), f);
    unpack8<T>(*reinterpret_cast<const uint4*>(zr), g);
  }
  if (w != nullptr) {
    float ss = 0.f, wf[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) ss = fmaf(f[i], f[i], ss);
#pragma unroll
    for (int s = L / 2; s > 0; s >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, s);
    const float inv = rsqrtf(ss / (float)DIM + eps);
    unpack8<T>(*reinterpret_cast<const uint4*>(w + c), wf);
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = to_f(from_f<T>(f[i] * inv * wf[i])) * (g[i] / (1.f + expf(-g[i])));
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = f[i] / (1.f + expf(-g[i]));
  }
  if (live) *reinterpret_cast<uint4*>(out + r * DIM + c) = pack8<T>(f);
}

}  // namespace

int gated_head_norm(void* out, const void* o, const void* z, const void* w, int64_t tokens, int heads, int dim, int rep,
                    int64_t z_stride, int64_t z_group, float eps, int dtype, cudaStream_t stream) {
  if (dim != 64 && dim != 128 && dim != 256) return 1;
  auto wide = [](const void* at) { return (reinterpret_cast<uintptr_t>(at) & 15) == 0; };
  if (!wide(out) || !wide(o) || !wide(z) || (w != nullptr && !wide(w)) || z_stride % 8 || z_group % 8) return 2;
  const int64_t rows = tokens * heads;
  if (rows <= 0) return 0;
  const unsigned blocks = (unsigned)((rows + 256 / (dim / 8) - 1) / (256 / (dim / 8)));
#define GHN(T, D)                                                                                                            \
  pdl_run(gated_head_norm_kernel<T, D>, blocks, 256, 0, stream, (T*)out, (const T*)o, (const T*)z, (const T*)w, rows, heads, rep, \
                                                           z_stride, z_group, eps)
  if (dtype == 0) {
    if (dim == 64) GHN(__nv_bfloat16, 64); else if (dim == 128) GHN(__nv_bfloat16, 128); else GHN(__nv_bfloat16, 256);
  } else {
    if (dim == 64) GHN(__half, 64); else if (dim == 128) GHN(__half, 128); else GHN(__half, 256);
  }
#undef GHN
  return 0;
}

int64_t gdn_scratch_bytes(int64_t tokens, int batch, int hq, int hv, int dtype) {
  return dtype == 0 ? gdn_max_chunks(tokens, batch) * hv * kChunkFloats * (int64_t)sizeof(float) : tokens * hq * (int64_t)sizeof(GdnLengths);
}

// Tokens up to which a sequence is faster a token at a time than in a chunk of 16 (or groups of four): a CTA's chain is a token's
// 1.4 us there and some 13 us for a chunk, behind the launch in front.  us by tokens / by chunks, 64 sequences of 32 heads, bf16:
// 2 tokens 66 / 101, 4 tokens 91 / 102, 5 tokens 103 / 103, 8 tokens 141 / 104; 4 sequences: 6 tokens 12.5 / 15.7, 8 tokens
// 14.4 / 15.5; fp16, by tokens / by groups, 64 sequences: 6 tokens 115 / 143, 8 tokens 140 / 145.
int gdn_short_len(int64_t sequences_by_heads, int dtype, int sms) { return dtype != 0 || sequences_by_heads <= sms ? 7 : 5; }

// Returns 0, or 1 when the head sizes are not 128 / the head counts do not divide.
int gdn_recurrent(const GdnParams& p, int dk, int dv, int dtype, cudaStream_t stream) {
  if (dk != kD || dv != kD || p.hq <= 0 || p.hv % p.hq != 0) return 1;
  if (p.batch <= 0 || p.tokens <= 0) return 0;
  if (dtype == 0) launch<__nv_bfloat16>(p, stream);
  else launch<__half>(p, stream);
  return 0;
}

}  // namespace b200
