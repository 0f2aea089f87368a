// Absorbed multi-head latent attention decode on tcgen05, dense, 16-bit latent cache.
//
//   q      [T, H, 576]   (q_nope . W_UK | q_pe), 16-bit
//   cache  [blocks, block_size, 576], same type; block_size a multiple of 32
//   out    [T, H, 512],  lse [H, T]
//
// The query tokens' visible cache rows, in tiles of 32, form one list, and groups of CTAs take equal contiguous ranges of it,
// whatever the lengths are.  A group covers 128 heads with two CTAs, one per HALF of the 512 latent output columns: the
// accumulator of 128 heads x 512 columns in fp32 is the whole tensor memory of an SM, which leaves no room for scores.  Both
// compute the (cheap to duplicate, 576-deep) score product; the second reader of a cache tile hits L2.  A range may end inside a
// token's list: such a part leaves its state (sums, maximum, denominator) in a slot, and the CTA that arrives last at the token
// adds the parts up when it is through with its range.  Nobody waits.
//
// Tensor memory of a CTA: S0 | S1 (32 fp32 columns each), O (256 columns), and the first 384 entries of its 128 query rows as
// packed 16-bit pairs (192 columns).  Only the other 192 entries stay in shared memory (48 KB), so that four cache tiles of 36 KB
// fit beside them and two thirds of the score product read no A operand from shared memory.
//
//   warp 4    TMA producer: cache tiles [32 x 576] through a 4-stage ring, one box per 64-wide chunk, without a break over the
//             ends of tokens; a tile never straddles a page, and the page of the next one is looked up ahead.  The query's last
//             three 64-wide chunks by TMA (heads beyond H are zero-filled by the tensor map).
//   warp 5    MMA issuer (one thread): S_j = Q . K_j^T (36 instructions of M128 N32 K16); O += P_j . V_j with P_j read from
//             tensor memory (it overwrites the first 16 columns of S_j as packed 16-bit pairs) and V_j = this CTA's 256 latent
//             columns of the SAME shared-memory tile, used in place as an MN-major operand (2 instructions of M128 N256 K16).
//             S_{j+1} is issued before P_j . V_j so the tensor core works while the softmax of tile j runs.
//   warps 0-3 softmax, thread = head: the query's first 384 entries to tensor memory; one tcgen05.ld brings the 32 scores of the
//             row, online softmax in the exp2 domain with a lazily moved maximum (the accumulator is rescaled in tensor memory
//             only when a row maximum grows by more than 2^8), P back with tcgen05.st; at a token's end the normalised output
//             half or the part and, from the CTA of half 0, the log-sum-exp.
//
// Rows of a token's last tile behind its visible length have P = 0 and are set to zero in shared memory, whatever the cache holds
// there.  Every wait is bounded; a wait that runs out records its site in the status word, the roles stop issuing and the CTA
// frees its tensor memory and returns.
//
// What bounds it: the chain of a tile (scores, softmax, product), the tensor core being half idle.  64 tokens of 128 heads, 256 to
// 4096 cached rows each: 347 us in the mma.sync kernel (mla_decode.cu; its query fragments are re-read from shared memory for every
// 8 rows) with three splits and a reduction behind it, 126 us here.
//
// Replaces flash_mla_with_kvcache (vllm_metax/v1/attention/backends/mla/flashmla.py:339-349) and the Triton split-KV
// MLA decode (vllm_metax/v1/attention/ops/triton_decode_attention.py:72-825) for ranks that hold 64 heads or more.
#include <type_traits>
#include "common.cuh"
#include "ptx_sm100.cuh"
#include "tma_host.h"
#include "ops.h"

namespace b200 {
using namespace ptx;

constexpr int kTcBM = 128;                       // head rows per CTA
constexpr int kTcBN = 32;                        // cache tokens per tile
constexpr int kTcD = 576, kTcDV = 512, kTcHalf = 256;
constexpr int kTcKC = kTcD / 64;                 // 64-wide chunks of a cache row
constexpr int kTcQT = 6;                         // of a query row, chunks in tensor memory; the others in shared memory
constexpr int kTcQChunk = kTcBM * 128;           // bytes of one 64-wide query chunk
constexpr int kTcKChunk = kTcBN * 128;           // bytes of one 64-wide cache chunk
constexpr int kTcQBytes = (kTcKC - kTcQT) * kTcQChunk;   // 49152
constexpr int kTcTileBytes = kTcKC * kTcKChunk;  // 36864
constexpr int kTcStages = 4;
constexpr int kTcMaxTokens = 1024;
constexpr int kTcShort = 4;                      // tiles of tokens that are not cut
constexpr int kTcSlot = kTcHalf * kTcBM + 2 * kTcBM;     // floats of a part: [64][128] float4, 128 maxima, 128 denominators
constexpr float kTcLazy = 8.f;                   // log2 of the growth of a row maximum that forces a rescale

struct TcSmem {
  static constexpr int kQ = 0;
  static constexpr int kKV = kQ + kTcQBytes;
  static constexpr int kBar = kKV + kTcStages * kTcTileBytes;
  static constexpr int kNumBars = 3 + 2 * kTcStages + 2 + 2 + 2 + 1;
  static constexpr int kPrefix = kBar + kNumBars * 8 + 16;
  static int dyn(int tokens) { return kPrefix + (tokens + 1) * 4 + 1024; }
};
static_assert(TcSmem::kPrefix + (kTcMaxTokens + 1) * 4 + 1024 <= 232448, "shared memory budget exceeded");

template <typename T>
__device__ __forceinline__ uint32_t tc_pack2(float a, float b);
template <>
__device__ __forceinline__ uint32_t tc_pack2<__nv_bfloat16>(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}
template <>
__device__ __forceinline__ uint32_t tc_pack2<__half>(float a, float b) {
  __half2 v = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float tc_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <typename T>
__global__ void __launch_bounds__(192, 1)
mla_decode_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmKV,
                     const MlaDecodeParams p, float* __restrict__ parts, int* __restrict__ counters) {
  using L = TcSmem;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kBar);
  uint64_t* q_full = bars;             // shared-memory part of a token's queries
  uint64_t* q_empty = bars + 1;        // the token's last score product has been formed
  uint64_t* qt_full = bars + 2;        // tensor-memory part
  uint64_t* kv_full = bars + 3;        // [4] stages
  uint64_t* kv_empty = kv_full + kTcStages;
  uint64_t* s_full = kv_empty + kTcStages;   // [2] score buffers
  uint64_t* p_full = s_full + 2;             // [2]
  uint64_t* o_done = p_full + 2;       // [2] of even and odd tiles (one alone could not tell the last from the one two before)
  uint64_t* met = o_done + 2;          // the softmax warps
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + L::kNumBars);
  int* s_pre = reinterpret_cast<int*>(smem + L::kPrefix);
  __shared__ int s_sum[6], s_max[6], s_done[2];

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int hf = blockIdx.x;                                  // latent half of the output
  const int h0 = blockIdx.y * kTcBM;
  const int T_ = p.total_tokens;

  constexpr uint32_t kTmemCols = 512;   // S0 [0,32) | S1 [32,64) | O [64,320) | Q [320,512)
  if (threadIdx.x == 0) {
    s_done[0] = s_done[1] = -1;
    mbar_init(q_full, 1);
    mbar_init(q_empty, 1);
    mbar_init(qt_full, 128);
    for (int i = 0; i < kTcStages; ++i) {
      mbar_init(&kv_full[i], 1);
      mbar_init(&kv_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[i], 128);
      mbar_init(&o_done[i], 1);
    }
    mbar_init(met, 128);
    fence_mbar_init();
    prefetch_tensormap(&tmQ);
    prefetch_tensormap(&tmKV);
  }
  if (warp == 5) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  // visible rows of token t (never past the block table) and its sequence
  auto visible = [&](int t, int& seq) -> int {
    int lo = 0, hi = p.batch - 1;
    if (p.query_start_loc) {                                  // the last b with query_start_loc[b] <= t
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (p.query_start_loc[mid] <= t) lo = mid; else hi = mid - 1;
      }
    } else {
      lo = t;
    }
    seq = lo;
    const int q0 = p.query_start_loc ? p.query_start_loc[lo] : lo;
    const int q1 = p.query_start_loc ? p.query_start_loc[lo + 1] : lo + 1;
    const long long cap = (long long)p.max_blocks * p.block_size;
    const int lim = p.seq_lens[lo] - (q1 - q0) + (t - q0) + 1;
    return lim > cap ? (int)cap : max(lim, 0);
  };
  // ---- tiles in front of every token (a token that sees nothing has one, all masked)
  {
    const int per = (T_ + 191) / 192;
    int sum = 0, seq, most = 0;
    for (int i = 0; i < per; ++i) {
      const int t = (int)threadIdx.x * per + i;
      if (t >= T_) break;
      const int n = max(1, (visible(t, seq) + kTcBN - 1) / kTcBN);
      s_pre[t + 1] = n;
      sum += n;
      most = max(most, n);
    }
    int inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += v;
      most = max(most, __shfl_xor_sync(0xffffffffu, most, o));
    }
    if (lane == 31) {
      s_sum[warp] = inc;
      s_max[warp] = most;
    }
    __syncthreads();
    int before = inc - sum;
    for (int w = 0; w < warp; ++w) before += s_sum[w];
    for (int i = 0; i < per; ++i) {
      const int t = (int)threadIdx.x * per + i;
      if (t >= T_) break;
      before += s_pre[t + 1];
      s_pre[t + 1] = before;
    }
    if (threadIdx.x == 0) s_pre[0] = 0;
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_S0 = tmem_base, tmem_S1 = tmem_base + 32, tmem_O = tmem_base + 64, tmem_Q = tmem_base + 320;
  const long long units = s_pre[T_];
  // groups: all there are, but a token's parts (1.5 us each to add up) no more than pays beside its tiles (0.8 us each)
  const int groups = (int)min(min((long long)gridDim.z, units),
                              (long long)T_ * max(1, (int)sqrtf(0.5f * (float)units / (float)T_)));
  const int grp = blockIdx.z;
  auto find = [&](int at) -> int {                            // the last token that starts at or before tile `at`
    int t = 0;
    for (int hi = T_ - 1; t < hi;) {
      const int mid = (t + hi + 1) >> 1;
      if (s_pre[mid] <= at) t = mid; else hi = mid - 1;
    }
    return t;
  };
  // ends of ranges; where all tokens are short, the nearer end of the token there: adding up parts would cost more than it saves
  const int longest = max(max(max(s_max[0], s_max[1]), max(s_max[2], s_max[3])), max(s_max[4], s_max[5]));
  auto border = [&](int c) -> int {
    const int at = (int)(units * c / groups);
    if (longest > kTcShort || c >= groups) return at;
    const int t = find(at);
    return at - s_pre[t] <= s_pre[t + 1] - at ? s_pre[t] : s_pre[t + 1];
  };
  const int u0 = grp < groups ? border(grp) : 0, u1 = grp < groups ? border(grp + 1) : 0;
  const int tok0 = find(u0);

  if (warp == 4) {
    // ------------------------------------------------------------ TMA producer
    if (lane == 0) {
      int g = 0, seg = 0;
      bool ok = true;
      for (int u = u0, t = tok0; u < u1 && ok; ++t, ++seg) {
        int seq;
        const int lim = visible(t, seq), first = u - s_pre[t], n = min(u1, s_pre[t + 1]) - u;
        const int* btab = p.block_table + (int64_t)seq * p.max_blocks;
        auto page_of = [&](int j) { return (first + j) * kTcBN < lim ? btab[(first + j) * kTcBN / p.block_size] : 0; };
        int next = page_of(0);
        for (int j = 0; j < n; ++j, ++g) {
          const int st = g % kTcStages;
          int page = next;
          if (j + 1 < n) next = page_of(j + 1);
          if (!mbar_wait(&kv_empty[st], ((g / kTcStages) & 1) ^ 1)) {
            report_status(p.status, kWaitTimeout, 60, j, st);
            ok = false;
            break;
          }
          if (page < 0 || page >= p.num_blocks) {
            report_status(p.status, kBadIndex, 61, (int)p.num_blocks, page);
            page = 0;
          }
          const int off = (first + j) * kTcBN % p.block_size;
          uint8_t* dst = smem + L::kKV + st * kTcTileBytes;
          mbar_expect_tx(&kv_full[st], kTcTileBytes);
#pragma unroll
          for (int c = 0; c < kTcKC; ++c) tma_load_3d(dst + c * kTcKChunk, &tmKV, &kv_full[st], c * 64, off, page);
          // the queries behind the first tiles, which need not wait for the token before
          if (j == min(n - 1, kTcStages - 2)) {
            if (!mbar_wait(q_empty, (seg & 1) ^ 1)) {
              report_status(p.status, kWaitTimeout, 68, j, st);
              ok = false;
              ++g;
              break;
            }
            mbar_expect_tx(q_full, kTcQBytes);
#pragma unroll
            for (int c = kTcQT; c < kTcKC; ++c)
              tma_load_3d(smem + L::kQ + (c - kTcQT) * kTcQChunk, &tmQ, q_full, c * 64, h0, t);
          }
        }
        if (!ok) break;
        u += n;
      }
      // no copy of this CTA is in flight when it returns: the last tiles have landed (immediate unless a role gave up before
      // consuming them), and so have the last queries
      for (int j = max(0, g - kTcStages); j < g; ++j) mbar_wait(&kv_full[j % kTcStages], (j / kTcStages) & 1);
      if (seg > 0) mbar_wait(q_full, (seg - 1) & 1);
    }
  } else if (warp == 5) {
    // ------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      constexpr uint32_t fmt = std::is_same<T, __half>::value ? 0u : 1u;
      constexpr uint32_t idesc_qk = make_idesc(1, fmt, fmt, kTcBM, kTcBN);
      // P.V: A = P from tensor memory (K-major), B = V in shared memory, MN-major (bit 16)
      constexpr uint32_t idesc_pv = make_idesc(1, fmt, fmt, kTcBM, kTcHalf) | (1u << 16);
      const uint32_t qa = smem_u32(smem + L::kQ);
      auto issue_qk = [&](int g, bool last) -> bool {
        const int st = g % kTcStages;
        if (!mbar_wait(&kv_full[st], (g / kTcStages) & 1)) {
          report_status(p.status, kWaitTimeout, 63, g, st);
          return false;
        }
        tc_fence_after_sync();
        const uint32_t ka = smem_u32(smem + L::kKV + st * kTcTileBytes);
        const uint32_t d = g & 1 ? tmem_S1 : tmem_S0;
#pragma unroll
        for (int c = 0; c < kTcQT; ++c) {
          const uint64_t dk = make_smem_desc_sw128(ka + c * kTcKChunk);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            umma_f16_ts(d, tmem_Q + c * 32 + k * 8, dk + (uint64_t)(k * 2), idesc_qk, (c | k) != 0 ? 1u : 0u);
        }
#pragma unroll
        for (int c = kTcQT; c < kTcKC; ++c) {
          const uint64_t dq = make_smem_desc_sw128(qa + (c - kTcQT) * kTcQChunk);
          const uint64_t dk = make_smem_desc_sw128(ka + c * kTcKChunk);
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_f16_ss(d, dq + (uint64_t)(k * 2), dk + (uint64_t)(k * 2), idesc_qk, 1u);
        }
        umma_commit(&s_full[g & 1]);
        if (last) umma_commit(q_empty);
        return true;
      };
      int g = 0, seg = 0;
      bool ok = true;
      for (int u = u0, t = tok0; u < u1 && ok; ++t, ++seg) {
        const int n = min(u1, s_pre[t + 1]) - u;
        if (!mbar_wait(qt_full, seg & 1) || !mbar_wait(q_full, seg & 1)) {
          report_status(p.status, kWaitTimeout, 62, seg, 0);
          break;
        }
        tc_fence_after_sync();
        ok = issue_qk(g, n == 1);
        for (int j = 0; j < n && ok; ++j, ++g) {
          const int st = g % kTcStages, sb = g & 1;
          if (j + 1 < n) {
            ok = issue_qk(g + 1, j + 2 == n);
            if (!ok) break;
          }
          if (!mbar_wait(&p_full[sb], (g >> 1) & 1)) {
            report_status(p.status, kWaitTimeout, 64, j, st);
            ok = false;
            break;
          }
          tc_fence_after_sync();
          // this CTA's 256 latent columns = chunks 4 hf .. 4 hf + 3 of the tile; contraction over 32 tokens in two steps
          const uint32_t va = smem_u32(smem + L::kKV + st * kTcTileBytes) + hf * 4 * kTcKChunk;
#pragma unroll
          for (int kk = 0; kk < kTcBN / 16; ++kk) {
            const uint64_t dv = make_smem_desc_sw128_mn(va + kk * 16 * 128, kTcKChunk);
            umma_f16_ts(tmem_O, (sb ? tmem_S1 : tmem_S0) + kk * 8, dv, idesc_pv, (j | kk) != 0 ? 1u : 0u);
          }
          umma_commit(&o_done[sb]);
          umma_commit(&kv_empty[st]);
        }
        u += n;
      }
    }
  } else {
    // ------------------------------------------------------------ softmax / output (warps 0..3), thread = head
    const int r = warp * 32 + lane;
    const int h = h0 + r;
    const bool row_valid = h < p.num_heads;
    const float sl2 = p.scale * 1.4426950408889634f;
    const uint32_t lane_base = ((uint32_t)(warp * 32)) << 16;
    // the first 384 entries of the row's query to tensor memory
    auto load_q = [&](int t) {
      const T* q = reinterpret_cast<const T*>(p.q) + (int64_t)t * p.q_stride + (int64_t)h * kTcD;
#pragma unroll 2
      for (int c = 0; c < kTcQT; ++c) {
        uint32_t v[32];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const uint4 x = row_valid ? *reinterpret_cast<const uint4*>(q + c * 64 + i * 8) : make_uint4(0u, 0u, 0u, 0u);
          v[4 * i] = x.x; v[4 * i + 1] = x.y; v[4 * i + 2] = x.z; v[4 * i + 3] = x.w;
        }
        tmem_st_32x32b_x32(tmem_Q + lane_base + c * 32, v);
      }
      tmem_st_wait();
      tc_fence_before_sync();
      mbar_arrive(qt_full);
    };
    // 32 columns from c on of the row's result
    auto store16 = [&](int t, int c, const float (&f)[32], float inv) {
      T* dst = reinterpret_cast<T*>(p.out) + ((int64_t)t * p.num_heads + h) * kTcDV + hf * kTcHalf + c;
#pragma unroll
      for (int g8 = 0; g8 < 4; ++g8) {
        float x[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = f[g8 * 8 + i] * inv;
        *reinterpret_cast<uint4*>(dst + g8 * 8) = pack8<T>(x);
      }
    };
    auto store_lse = [&](int t, float m, float l) {
      if (hf == 0 && p.lse_out) p.lse_out[(int64_t)h * T_ + t] = l > 0.f ? m * 0.6931471805599453f + logf(l) : -INFINITY;
    };
    // the groups that hold a token's tiles; where a group leaves its part of one: its range starts inside the token, or not
    auto sharers = [&](int t, int& c0, int& c1) {
      c0 = (int)(((long long)s_pre[t] * groups + groups - 1) / units);
      c1 = (int)(((long long)s_pre[t + 1] * groups - 1) / units);
    };
    auto slot = [&](int c, bool tail) {
      return parts + ((((int64_t)c * gridDim.y + blockIdx.y) * 2 + hf) * 2 + (tail ? 0 : 1)) * kTcSlot;
    };
    // (a bounded wait, too: a warp that gave up does not come)
    int meetings = 0;
    auto meet = [&]() -> bool {
      mbar_arrive(met);
      return __all_sync(0xffffffffu, mbar_wait(met, meetings++ & 1));
    };
    bool ok = true;
    int g = 0;
    if (u0 < u1) load_q(tok0);
    for (int u = u0, t = tok0; u < u1 && ok; ++t) {
      int seq;
      const int lim = visible(t, seq), first = u - s_pre[t], end = min(u1, s_pre[t + 1]), n = end - u;
      float m_run = -INFINITY, l_run = 0.f;
      for (int j = 0; j < n; ++j, ++g) {
        const int st = g & 1;
        // (every give-up decision is taken by the whole warp: the tensor-memory loads below are warp-collective)
        if (!__all_sync(0xffffffffu, mbar_wait(&s_full[st], (g >> 1) & 1))) {
          report_status(p.status, kWaitTimeout, 65, j, st);
          ok = false;
          break;
        }
        tc_fence_after_sync();
        const uint32_t tmem_St = (st ? tmem_S1 : tmem_S0) + lane_base;
        uint32_t sv[32];
        tmem_ld_32x32b_x32(tmem_St, sv);
        tmem_ld_wait();
        float s[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) s[i] = __uint_as_float(sv[i]) * sl2;
        const int row0 = (first + j) * kTcBN;
        if (row0 + kTcBN > lim) {
          // rows that nobody sees: no weight, and zeros for what the cache may hold there
          const int seen = max(0, lim - row0);
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (i >= seen) s[i] = -INFINITY;
          uint8_t* v = smem + L::kKV + g % kTcStages * kTcTileBytes + hf * 4 * kTcKChunk;
          for (int i = r; i < (kTcBN - seen) * 32; i += 128) {
            const int row = seen + i / 32, c = i % 32;
            *reinterpret_cast<uint4*>(v + (c / 8) * kTcKChunk + row * 128 + (c % 8) * 16) = make_uint4(0u, 0u, 0u, 0u);
          }
          fence_proxy_async();
        }
        float mx = s[0];
#pragma unroll
        for (int i = 1; i < 32; ++i) mx = fmaxf(mx, s[i]);
        const bool grow = mx > m_run + kTcLazy;        // also true for the first finite maximum
        float corr = 1.f;
        if (grow) {
          corr = (m_run == -INFINITY) ? 0.f : exp2f(m_run - mx);
          m_run = mx;
          l_run *= corr;
        }
        if (j > 0 && __any_sync(0xffffffffu, grow)) {
          // the product of tile j - 1 must have landed before the accumulator is rescaled
          if (!__all_sync(0xffffffffu, mbar_wait(&o_done[(g - 1) & 1], ((g - 1) >> 1) & 1))) {
            report_status(p.status, kWaitTimeout, 66, j, st);
            ok = false;
            break;
          }
          tc_fence_after_sync();
#pragma unroll 1
          for (int c = 0; c < kTcHalf; c += 32) {
            uint32_t v[32];
            tmem_ld_32x32b_x32(tmem_O + lane_base + c, v);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * corr);
            tmem_st_32x32b_x32(tmem_O + lane_base + c, v);
          }
        }
        const float m_off = (m_run == -INFINITY) ? 0.f : m_run;
        float rs = 0.f;
        uint32_t pk[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float e0 = tc_exp2(s[2 * i] - m_off);
          const float e1 = tc_exp2(s[2 * i + 1] - m_off);
          rs += e0 + e1;
          pk[i] = tc_pack2<T>(e0, e1);
        }
        tmem_st_32x32b_x16(tmem_St, pk);
        l_run += rs;
        // P (and a rescaled accumulator) visible to the MMA warp
        tmem_st_wait();
        tc_fence_before_sync();
        mbar_arrive(&p_full[st]);
      }
      if (!ok) break;
      if (end < u1) load_q(t + 1);                     // (all score products of this token have been formed)
      if (!__all_sync(0xffffffffu, mbar_wait(&o_done[(g - 1) & 1], ((g - 1) >> 1) & 1))) {
        report_status(p.status, kWaitTimeout, 67, n, 0);
        ok = false;
        break;
      }
      tc_fence_after_sync();
      const bool tail = first != 0, whole = !tail && end == s_pre[t + 1];
      const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
      float* mine = slot(grp, tail);
#pragma unroll 1
      for (int c = 0; c < kTcHalf; c += 32) {
        uint32_t v[32];
        tmem_ld_32x32b_x32(tmem_O + lane_base + c, v);
        tmem_ld_wait();
        float f[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) f[i] = __uint_as_float(v[i]);
        if (whole) {
          if (row_valid) store16(t, c, f, inv);
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i)
            reinterpret_cast<float4*>(mine)[(c / 4 + i) * kTcBM + r] = make_float4(f[4 * i], f[4 * i + 1], f[4 * i + 2], f[4 * i + 3]);
        }
      }
      if (whole) {
        if (row_valid) store_lse(t, m_run, l_run);
      } else {
        mine[kTcHalf * kTcBM + r] = m_run;
        mine[kTcHalf * kTcBM + kTcBM + r] = l_run;
        __threadfence();
        if (!meet()) {
          report_status(p.status, kWaitTimeout, 69, n, 0);
          ok = false;
          break;
        }
        if (threadIdx.x == 0) {
          int c0, c1;
          sharers(t, c0, c1);
          const bool last = atomicAdd(&counters[(t * (int)gridDim.y + blockIdx.y) * 2 + hf], 1) == c1 - c0;
          s_done[tail ? 0 : 1] = last ? t : -1;
        }
      }
      u = end;
    }
    // tokens whose last part was one of this CTA's (at most its first and its last)
    if (ok) ok = meet();
#pragma unroll 1
    for (int i = 0; ok && i < 2; ++i) {
      const int t = s_done[i];
      if (t < 0) continue;
      __threadfence();
      int c0, c1;
      sharers(t, c0, c1);
      const bool tail0 = units * c0 / groups > s_pre[t];
      float M = -INFINITY, l = 0.f;
      for (int c = c0; c <= c1; ++c) M = fmaxf(M, __ldcg(slot(c, c > c0 || tail0) + kTcHalf * kTcBM + r));
      const float ms = M == -INFINITY ? 0.f : M;
      for (int c = c0; c <= c1; ++c) {
        const float* at = slot(c, c > c0 || tail0) + kTcHalf * kTcBM + r;
        l += __ldcg(at + kTcBM) * exp2f(__ldcg(at) - ms);
      }
      const float inv = l > 0.f ? 1.f / l : 0.f;
#pragma unroll 1
      for (int col = 0; col < kTcHalf; col += 32) {
        float f[32];
#pragma unroll
        for (int e = 0; e < 32; ++e) f[e] = 0.f;
#pragma unroll 2
        for (int c = c0; c <= c1; ++c) {
          const float* at = slot(c, c > c0 || tail0);
          const float w = exp2f(__ldcg(at + kTcHalf * kTcBM + r) - ms);
          float4 x[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) x[e] = __ldcg(reinterpret_cast<const float4*>(at) + (col / 4 + e) * kTcBM + r);
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            f[4 * e] = fmaf(x[e].x, w, f[4 * e]); f[4 * e + 1] = fmaf(x[e].y, w, f[4 * e + 1]);
            f[4 * e + 2] = fmaf(x[e].z, w, f[4 * e + 2]); f[4 * e + 3] = fmaf(x[e].w, w, f[4 * e + 3]);
          }
        }
        if (row_valid) store16(t, col, f, inv);
      }
      if (row_valid) store_lse(t, ms, l);
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 5) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

static int tc_groups(const MlaDecodeParams& p, int sms) {
  const int tiles = (p.num_heads + kTcBM - 1) / kTcBM, g = sms / (2 * tiles);
  return g > 1 ? g : 1;
}

// Whether the kernel serves the call: dense, DeepSeek sizes, no window, a block size that is a multiple of 32, aligned operands.
bool mla_decode_tc_serves(const MlaDecodeParams& p) {
  return p.topk_indices == nullptr && p.window <= 0 && p.kv_rank == kTcDV && p.q_dim == kTcD && p.row_elems == kTcD &&
         p.total_tokens <= kTcMaxTokens && p.block_size % kTcBN == 0 && p.max_blocks > 0 && p.num_blocks > 0 &&
         (reinterpret_cast<uintptr_t>(p.q) & 15) == 0 && p.q_stride % 8 == 0 && (reinterpret_cast<uintptr_t>(p.cache) & 15) == 0 &&
         (reinterpret_cast<uintptr_t>(p.out) & 15) == 0;
}

// Scratch: *floats of parts, *ints of counters, which are zero.
void mla_decode_tc_scratch(const MlaDecodeParams& p, int sms, int64_t* floats, int64_t* ints) {
  const int tiles = (p.num_heads + kTcBM - 1) / kTcBM;
  *floats = (int64_t)tc_groups(p, sms) * tiles * 4 * kTcSlot;
  *ints = (int64_t)p.total_tokens * tiles * 2;
}

void mla_decode_tc(const MlaDecodeParams& p, int dtype, int sms, float* parts, int* counters, cudaStream_t stream) {
  const CUtensorMapDataType dt = dtype == 1 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  // q: [T, H, 576] -> dims (576, H, T), box (64, 128 heads, 1 token)
  uint64_t qd[3] = {(uint64_t)kTcD, (uint64_t)p.num_heads, (uint64_t)p.total_tokens};
  uint64_t qs[2] = {(uint64_t)kTcD * 2, (uint64_t)p.q_stride * 2};
  uint32_t qb[3] = {64, (uint32_t)kTcBM, 1};
  const CUtensorMap tmQ = make_tmap_nd(p.q, dt, 3, qd, qs, qb, CU_TENSOR_MAP_SWIZZLE_128B);
  // cache: [blocks, block_size, 576] -> dims (576, block_size, blocks), box (64, 32 tokens, 1 page)
  uint64_t kd[3] = {(uint64_t)kTcD, (uint64_t)p.block_size, (uint64_t)p.num_blocks};
  uint64_t ks[2] = {(uint64_t)kTcD * 2, (uint64_t)p.block_size * kTcD * 2};
  uint32_t kb[3] = {64, (uint32_t)kTcBN, 1};
  const CUtensorMap tmKV = make_tmap_nd(p.cache, dt, 3, kd, ks, kb, CU_TENSOR_MAP_SWIZZLE_128B);
  const dim3 grid(2, (unsigned)((p.num_heads + kTcBM - 1) / kTcBM), (unsigned)tc_groups(p, sms));
  const int bytes = TcSmem::dyn(p.total_tokens);
  if (dtype == 1) {
    auto kern = mla_decode_tc_kernel<__half>;
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    kern<<<grid, 192, bytes, stream>>>(tmQ, tmKV, p, parts, counters);
  } else {
    auto kern = mla_decode_tc_kernel<__nv_bfloat16>;
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    kern<<<grid, 192, bytes, stream>>>(tmQ, tmKV, p, parts, counters);
  }
}

}  // namespace b200
