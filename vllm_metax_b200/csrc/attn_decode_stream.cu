// Paged GQA decode attention, one token per sequence, with the KV stream shared out evenly whatever the lengths are.
//
// The sequences' tokens, in units of 64, form one list, with two units more for the end of each (without these, a step's many short
// rows, such as those that pad a captured one, came to one CTA); the CTAs of a key head (as many as fit on the GPU at once) take
// equal contiguous ranges of it, and neighbouring CTAs the same range of neighbouring heads, whose rows lie side by side in a page.  A
// range may end inside a sequence: such a part leaves its state (sums, maximum, denominator) in a slot, and the CTA that arrives
// last at the sequence adds the parts up when it is through with its range, all its warps at once.  Nobody waits.  A CTA copies
// without a break from its first unit to its last: the ring of tiles runs on over the ends of sequences, the page of a tile is
// looked up one tile ahead, and the next sequence's queries arrive while this one is computed.
//
// Each of 4 warps owns a quarter of every unit (16 tokens) and runs the flash recurrence with m16n8k16 products on the rows of its
// heads; the four states meet in shared memory at a sequence's end.  ROWS: heads per key head, 8 or 16; with 8 the lower half of
// the product's rows does not exist for the softmax.
//
// int8 caches (KIND 1, one scale per token and head): tiles stay bytes in shared memory and become 16-bit operands in registers.
// The contraction over a head's entries runs in the order in which a lane finds them - lane t of four owns the 32 bytes from 32 t
// on - and value columns likewise (lane g the 16 bytes from 16 g on), so fragments are 16-byte loads and byte permutations; the
// integers are exact in either 16-bit type.
//
// What bounds it: the KV bytes; with few or ragged rows the ends of ranges and of sequences.  One CTA per (sequence, head) and
// tiles converted through shared memory / now, us:
//   256 rows of 1088 tokens, 32 heads over 8, bf16      234 / 190   (its bytes at copy bandwidth: 177)
//   16 rows, 64 heads over 8, int8                       472 / 208   (91)
//   64 rows, 32 heads over 4, bf16                        51 / 35
//   64 rows of 2 key heads of 256, bf16                   81 / 56
//   40 rows of 42 thousand tokens in all and 8 that pad, 32 over 8   54 / 47   (58 before ends counted in the ranges)
//   100 rows of 37 thousand tokens and 12 that pad        58 / 49   (65)
//   1 row of 900                                          13 / 13
//   32 rows of 128, 32 over 8                             12 / 17   (a sequence's parts; such steps are where it loses)
// Covers the same calls as attn_decode.cu (see there for the reference's).
#include <type_traits>
#include "attn_decode.cuh"
#include "attn_score.cuh"
#include "ops.h"
#include "pdl.cuh"

namespace b200 {
namespace {

constexpr int kWarps = 4, kThreads = 128, kTile = 16, kStages = 3, kMaxBatch = 1024, kMaxSmem = 227 * 1024;
constexpr int kEnd = 2;                                                   // what a sequence's end costs a CTA, in units
constexpr float kLog2e = 1.4426950408889634f, kLn2 = 0.6931471805599453f;

template <int D, int KIND, int ROWS>
struct StreamSmem {
  static constexpr int kRow = KIND == 0 ? D * 2 : D;                      // bytes of a tile's row
  static constexpr int kTileBytes = kTile * kRow;
  static constexpr int kStage = 2 * kTileBytes + (KIND == 0 ? 0 : 2 * kTile * 4);
  static constexpr int kQ = 0, kQBytes = ROWS * D * 2;                    // two of them
  static constexpr int kRing = 2 * kQBytes;
  static constexpr int kMerge = kRing + kWarps * kStages * kStage;        // two states
  static constexpr int kState = ROWS * D * 4 + 2 * ROWS * 4;
  static constexpr int kPrefix = kMerge + 2 * kState;
  static int total(int batch) { return kPrefix + (batch + 1) * 4; }
};

// Bytes j of two words as 16-bit integers' values: int8 is exact in both types.
//   fp16: 1024 + (b + 128) is 0x6400 | (b ^ 0x80); minus 1152.
//   bf16: 128 + (b & 127) is 0x4300 | (b & 0x7f), and 0x4300 | (b & 0x80) is 128 or, for negative b, 256; the difference.
template <typename T>
__device__ __forceinline__ uint32_t widen(uint32_t t) {                   // (the upper byte of either half is arbitrary)
  if constexpr (std::is_same<T, __half>::value) {
    const uint32_t x = ((t & 0x00ff00ffu) ^ 0x00800080u) | 0x64006400u;
    const __half2 r = __hsub2(*reinterpret_cast<const __half2*>(&x), __floats2half2_rn(1152.f, 1152.f));
    return *reinterpret_cast<const uint32_t*>(&r);
  } else {
    const uint32_t x = (t & 0x007f007fu) | 0x43004300u, c = (t & 0x00800080u) | 0x43004300u;
    const __nv_bfloat162 r = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&x), *reinterpret_cast<const __nv_bfloat162*>(&c));
    return *reinterpret_cast<const uint32_t*>(&r);
  }
}

template <typename T, int D, int KIND, int ROWS>
__global__ void __launch_bounds__(kThreads, (D > 128 ? 1 : KIND == 1 ? 3 : 2))
paged_decode_stream_kernel(const DecodeParams p, int batch, float* parts, int* counters) {
  using S = StreamSmem<D, KIND, ROWS>;
  constexpr int CPR = D / 8, ND = D / 8;
  extern __shared__ __align__(128) uint8_t smem[];
  pdl_trigger();
  pdl_wait();
  __shared__ int s_sum[kWarps], s_done[2];
  if (threadIdx.x < 2) s_done[threadIdx.x] = -1;
  int* s_pre = reinterpret_cast<int*>(smem + S::kPrefix);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = p.num_q_heads / p.num_kv_heads;
  const int hk = blockIdx.x % p.num_kv_heads, grp = blockIdx.x / p.num_kv_heads;
  const int dqk = KIND == 0 ? p.dqk : D, dv = KIND == 0 ? p.dv : D;
  const long long kv_cap = (long long)p.max_blocks * p.block_size;

  // length, first visible tile and units of a sequence; a length the block table cannot hold is recorded and cut
  auto extent = [&](int b, int& kv_len, int& tile_lo) -> int {
    kv_len = p.seq_lens[b];
    if (kv_len < 0 || kv_len > kv_cap) {
      report_status(p.status, kBadIndex, 21, (int)(kv_cap > 0x7fffffff ? 0x7fffffff : kv_cap), kv_len);
      kv_len = kv_len < 0 ? 0 : (int)kv_cap;
    }
    tile_lo = first_key(kv_len, p.window, p.chunk) / kTile;
    return max(1, ((kv_len + kTile - 1) / kTile - tile_lo + kWarps - 1) / kWarps);
  };
  // ---- what is in front of every sequence: units, and kEnd for the end of each
  {
    const int per = (batch + kThreads - 1) / kThreads;
    int sum = 0, x, y;
    for (int i = 0; i < per; ++i) {
      const int b = tid * per + i;
      if (b >= batch) break;
      const int n = extent(b, x, y) + kEnd;
      s_pre[b + 1] = n;
      sum += n;
    }
    int inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += v;
    }
    if (lane == 31) s_sum[warp] = inc;
    __syncthreads();
    int before = inc - sum;
    for (int w = 0; w < warp; ++w) before += s_sum[w];
    for (int i = 0; i < per; ++i) {
      const int b = tid * per + i;
      if (b >= batch) break;
      before += s_pre[b + 1];
      s_pre[b + 1] = before;
    }
    if (tid == 0) s_pre[0] = 0;
    __syncthreads();
  }
  const long long space = s_pre[batch];
  // every range holds a unit; and a sequence's parts, which one CTA adds up, are no more than pays beside its units
  const long long units = space - (long long)kEnd * batch;
  const int groups = (int)min(min((long long)(gridDim.x / p.num_kv_heads), units),
                              (long long)batch * max(1, (int)sqrtf(4.f * (float)units / (float)batch)));
  if (grp >= groups) return;
  // where range c begins: a unit of sequence `seq`, in units and ends from the first one on
  auto border = [&](int c, int& seq) -> int {
    const int at = (int)(space * c / groups);
    int lo = 0;
    for (int hi = batch; lo < hi;) {                                      // the last sequence that starts at or before `at`
      const int mid = (lo + hi + 1) >> 1;
      if (s_pre[mid] <= at) lo = mid; else hi = mid - 1;
    }
    seq = lo;
    if (lo == batch || at < s_pre[lo + 1] - kEnd) return at;
    return s_pre[seq = lo + 1];                                           // (within its end: the next one)
  };
  int b, b_end;
  const int u0 = border(grp, b), u1 = border(grp + 1, b_end);
  if (u0 >= u1) return;

  uint8_t* ring = smem + S::kRing + warp * kStages * S::kStage;
  // queries of sequence `seq` into buffer `qb`: 16-byte chunks, swizzled for ldmatrix (16-bit caches) or as they are
  auto copy_q = [&](int seq, int qb) {
    const T* src = reinterpret_cast<const T*>(p.q) + (int64_t)seq * p.q_stride + (int64_t)hk * g * dqk;
    for (int i = tid; i < g * CPR; i += kThreads) {
      const int r = i / CPR, c = i % CPR;
      const bool ok = c * 8 < dqk;
      uint8_t* dst = smem + S::kQ + qb * S::kQBytes + r * D * 2 + (KIND == 0 ? (c ^ (r & 7)) : c) * 16;
      cp_async16(dst, ok ? src + (int64_t)r * dqk + c * 8 : reinterpret_cast<const T*>(p.q), ok);
    }
  };

  // ---- what is copied next: tile `warp` of unit iu of sequence ib
  int ib = b, iu = u0 - s_pre[b], in, ilen, itile_lo, ileft = u1 - u0 - kEnd * (b_end - b), ipage = -1;
  in = extent(ib, ilen, itile_lo);
  auto look_up = [&]() {
    const int tok0 = (itile_lo + iu * kWarps + warp) * kTile;
    ipage = -1;
    if (ileft > 0 && tok0 < ilen) ipage = p.block_table[(int64_t)ib * p.max_blocks + tok0 / p.block_size];
  };
  look_up();
  auto issue = [&](int stage) {
    const int tok0 = (itile_lo + iu * kWarps + warp) * kTile;
    if (ileft > 0 && tok0 < ilen) {
      int page = ipage;
      if (page < 0 || page >= p.num_blocks) {
        report_status(p.status, kBadIndex, 20, (int)p.num_blocks, page);
        page = 0;
      }
      const int off0 = tok0 % p.block_size;
      uint8_t* st = ring + stage * S::kStage;
      constexpr int RC = S::kRow / 16, kElem = KIND == 0 ? 2 : 1;
#pragma unroll
      for (int kv = 0; kv < 2; ++kv) {
        const uint8_t* cache = reinterpret_cast<const uint8_t*>(kv ? p.v_cache : p.k_cache);
        const int d = kv ? dv : dqk;
        const uint8_t* rows = cache + ((int64_t)page * p.page_stride + ((int64_t)off0 * p.num_kv_heads + hk) * d) * kElem;
        const int64_t row_bytes = (int64_t)p.num_kv_heads * d * kElem;
#pragma unroll
        for (int i = 0; i < kTile * RC / 32; ++i) {
          const int idx = lane + i * 32, r = idx / RC, c = idx % RC;
          const bool ok = tok0 + r < ilen && (KIND != 0 || c * 8 < d);
          const int dc = KIND == 0 ? (c ^ (r & 7)) : kv ? (c ^ (((r >> 1) & 3) << 1)) : (c ^ (r & 1));
          cp_async16(st + kv * S::kTileBytes + r * S::kRow + dc * 16, ok ? rows + r * row_bytes + c * 16 : cache, ok);
        }
        if constexpr (KIND != 0) {
          if (lane < kTile) {
            const bool ok = tok0 + lane < ilen;
            const float* src = p.kv_scales + (((int64_t)page * 2 + kv) * p.block_size + off0 + lane) * p.num_kv_heads + hk;
            cp_async4(st + 2 * S::kTileBytes + (kv * kTile + lane) * 4, ok ? src : p.kv_scales, ok);
          }
        }
      }
    }
    --ileft;
    if (++iu == in && ileft > 0) {
      iu = 0;
      in = extent(++ib, ilen, itile_lo);
    }
    look_up();
  };

  // ---- rows of this lane: ra, and with 16 rows rb
  const int ra = lane >> 2, rb = ra + 8, tl = lane & 3;
  constexpr int H = ROWS / 8;
  const bool live[2] = {ra < g, H > 1 && rb < g};
  float al[2], sh[2], far[2];
  const float* bs[2];
  const bool sigmoid = p.sigmoid_shift != nullptr;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int hq = hk * g + (h ? rb : ra);
    al[h] = p.alibi_slopes && live[h] ? p.alibi_slopes[hq] * kLog2e : 0.f;
    sh[h] = sigmoid && live[h] ? p.sigmoid_shift[hq] * kLog2e : 0.f;
    bs[h] = p.bias && live[h] ? p.bias + (int64_t)hq * p.bias_len : nullptr;
    far[h] = bs[h] ? bs[h][p.bias_len - 1] * kLog2e : 0.f;
  }
  const float scale2 = p.scale * kLog2e, m_start = sigmoid ? 0.f : -INFINITY;
  float m[2], l[2], o[ND][4];
  auto clear = [&]() {
#pragma unroll
    for (int h = 0; h < 2; ++h) { m[h] = m_start; l[h] = 0.f; }
#pragma unroll
    for (int i = 0; i < ND; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
  };
  // a state in memory: [H][ND][32] pairs, then [2][ROWS] maxima and denominators
  auto put = [&](float* at) {
#pragma unroll
    for (int h = 0; h < H; ++h) {
#pragma unroll
      for (int i = 0; i < ND; ++i)
        *reinterpret_cast<float2*>(at + ((h * ND + i) * 32 + lane) * 2) = make_float2(o[i][2 * h], o[i][2 * h + 1]);
      if (tl == 0) {
        at[ROWS * D + (h ? rb : ra)] = m[h];
        at[ROWS * D + ROWS + (h ? rb : ra)] = l[h];
      }
    }
  };
  auto add = [&](const float* at) {
#pragma unroll
    for (int h = 0; h < H; ++h) {
      float2 x[ND];
#pragma unroll
      for (int i = 0; i < ND; ++i) x[i] = *reinterpret_cast<const float2*>(at + ((h * ND + i) * 32 + lane) * 2);
      const float mo = at[ROWS * D + (h ? rb : ra)], lo = at[ROWS * D + ROWS + (h ? rb : ra)];
      const float mn = fmaxf(m[h], mo), ms = mn == -INFINITY ? 0.f : mn;
      const float f0 = exp2f(m[h] - ms), f1 = exp2f(mo - ms);
      m[h] = mn;
      l[h] = l[h] * f0 + lo * f1;
#pragma unroll
      for (int i = 0; i < ND; ++i) {
        o[i][2 * h] = o[i][2 * h] * f0 + x[i].x * f1;
        o[i][2 * h + 1] = o[i][2 * h + 1] * f0 + x[i].y * f1;
      }
    }
  };
  float* merge[2] = {reinterpret_cast<float*>(smem + S::kMerge), reinterpret_cast<float*>(smem + S::kMerge + S::kState)};
  // The result of sequence `seq` from n states, the i-th `step` floats behind the first but for the last one, at `end`.  Several
  // states are on their way at a time; their weights refer to the largest maximum among them.
  auto write = [&](int seq, int n, const float* at, int64_t step, const float* end) {
    constexpr int K = ND / 4, B = D > 128 ? 4 : 8;
    const int64_t out_stride = p.out_stride ? p.out_stride : (int64_t)p.num_q_heads * dv;
#pragma unroll 1
    for (int h = 0; h < H; ++h) {
      const int r = h ? rb : ra, hq = hk * g + r;
      float M = -INFINITY, L = 0.f;
      float2 acc[K];
#pragma unroll
      for (int k = 0; k < K; ++k) acc[k] = make_float2(0.f, 0.f);
#pragma unroll 1
      for (int j = 0; j < n; j += B) {
        float mo[B], lo[B];
        float2 v[B][K];
#pragma unroll
        for (int i = 0; i < B; ++i) {
          mo[i] = -INFINITY;
          lo[i] = 0.f;
#pragma unroll
          for (int k = 0; k < K; ++k) v[i][k] = make_float2(0.f, 0.f);
          if (j + i < n) {
            const float* x = j + i + 1 == n ? end : at + (j + i) * step;
            mo[i] = x[ROWS * D + r];
            lo[i] = x[ROWS * D + ROWS + r];
#pragma unroll
            for (int k = 0; k < K; ++k) v[i][k] = *reinterpret_cast<const float2*>(x + ((h * ND + warp + 4 * k) * 32 + lane) * 2);
          }
        }
        float mn = M;
#pragma unroll
        for (int i = 0; i < B; ++i) mn = fmaxf(mn, mo[i]);
        const float s = mn == -INFINITY ? 0.f : mn, f0 = exp2f(M - s);
        M = mn;
        L *= f0;
#pragma unroll
        for (int k = 0; k < K; ++k) { acc[k].x *= f0; acc[k].y *= f0; }
#pragma unroll
        for (int i = 0; i < B; ++i) {
          const float f1 = exp2f(mo[i] - s);
          L = fmaf(lo[i], f1, L);
#pragma unroll
          for (int k = 0; k < K; ++k) {
            acc[k].x = fmaf(v[i][k].x, f1, acc[k].x);
            acc[k].y = fmaf(v[i][k].y, f1, acc[k].y);
          }
        }
      }
      if (r >= g) continue;
      const float ms = M == -INFINITY ? 0.f : M;
      if (sigmoid) L = 1.f;
      if (p.sinks) L += exp2f(p.sinks[hq] * kLog2e - ms);
      const float inv = L > 0.f ? p.out_scale / L : 0.f;
      T* out = reinterpret_cast<T*>(p.out) + seq * out_stride + (int64_t)hq * dv;
      const int64_t gt = seq * p.gate_stride + (p.gate_per_head ? hq : (int64_t)hq * dv);
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const int nd = warp + 4 * k, c0 = KIND == 0 ? nd * 8 + 2 * tl : 2 * tl * (D / 8) + nd, c1 = KIND == 0 ? c0 + 1 : c0 + D / 8;
        if (c0 < dv) out[c0] = from_f<T>(acc[k].x * inv * gate_of<T>(p.gate, gt + (p.gate_per_head ? 0 : c0)));
        if (c1 < dv) out[c1] = from_f<T>(acc[k].y * inv * gate_of<T>(p.gate, gt + (p.gate_per_head ? 0 : c1)));
      }
      if (p.lse_out && warp == 0 && tl == 0) p.lse_out[(int64_t)hq * p.total_tokens + seq] = L > 0.f ? ms * kLn2 + logf(L) : -INFINITY;
    }
  };
  // the CTAs that hold a sequence's units, and where a CTA leaves its part of one: a range that starts inside the sequence, or not
  auto sharers = [&](int seq, int& c0, int& c1) {
    c0 = (int)(((long long)s_pre[seq] * groups + groups - 1) / space);
    c1 = (int)(((long long)(s_pre[seq + 1] - kEnd) * groups - 1) / space);
  };
  constexpr int kSlot = S::kState / 4;
  auto slot = [&](int c, bool tail) { return parts + (((int64_t)c * p.num_kv_heads + hk) * 2 + (tail ? 0 : 1)) * kSlot; };

  copy_q(b, 0);
#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) {
    issue(s);
    cp_async_commit();
  }
  cp_async_wait<kStages - 2>();                                           // (the queries are in the first group)
  __syncthreads();
  int stage = 0, qb = 0, u = u0, left0 = -1, left1 = -1;
  while (u < u1) {
    // ---- one sequence's share of this CTA: units u .. seg_end
    int kv_len, tile_lo;
    extent(b, kv_len, tile_lo);
    const int first = s_pre[b], behind = s_pre[b + 1] - kEnd, seg_end = min(u1, behind), seg0 = u;
    const int lo_pos = first_key(kv_len, p.window, p.chunk);
    clear();
    uint32_t qf[D / 16][4];
    {
      const uint8_t* qs = smem + S::kQ + qb * S::kQBytes;
      if constexpr (KIND == 0) {
        const int mat = lane >> 3, r = ((mat & 1) * 8 + (lane & 7)) & (ROWS - 1);
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) ldmatrix_x4(qf[ks], qs + r * D * 2 + (((2 * ks + (mat >> 1)) ^ (r & 7)) * 16));
      } else {
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
          const uint2 x = *reinterpret_cast<const uint2*>(qs + ra * D * 2 + (tl * (D / 4) + ks * 4) * 2);
          const uint2 y = *reinterpret_cast<const uint2*>(qs + (rb & (ROWS - 1)) * D * 2 + (tl * (D / 4) + ks * 4) * 2);
          qf[ks][0] = x.x; qf[ks][1] = y.x; qf[ks][2] = x.y; qf[ks][3] = y.y;
        }
      }
    }
    for (; u < seg_end; ++u) {
      issue((stage + kStages - 1) % kStages);
      if (u == seg0 && seg_end + kEnd < u1) copy_q(b + 1, qb ^ 1);
      cp_async_commit();
      cp_async_wait<kStages - 1>();
      __syncwarp();
      const int tok0 = (tile_lo + (u - first) * kWarps + warp) * kTile;
      if (tok0 < kv_len) {
        const uint8_t* st = ring + stage * S::kStage;
        const uint8_t *k_tile = st, *v_tile = st + S::kTileBytes;
        float s[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
        float ksc[4] = {1.f, 1.f, 1.f, 1.f}, vsc[4] = {1.f, 1.f, 1.f, 1.f};
        if constexpr (KIND == 0) {
#pragma unroll
          for (int ks = 0; ks < D / 16; ++ks) {
            uint32_t kf[4];
            const int mat = lane >> 3, r = (mat >> 1) * 8 + (lane & 7);
            ldmatrix_x4(kf, k_tile + r * S::kRow + (((2 * ks + (mat & 1)) ^ (r & 7)) * 16));
            mma16816<T>(s[0], qf[ks], kf[0], kf[1]);
            mma16816<T>(s[1], qf[ks], kf[2], kf[3]);
          }
        } else {
          const float* sc = reinterpret_cast<const float*>(st + 2 * S::kTileBytes);
          const int c0 = 2 * tl;
          ksc[0] = sc[c0]; ksc[1] = sc[c0 + 1]; ksc[2] = sc[8 + c0]; ksc[3] = sc[8 + c0 + 1];
          vsc[0] = sc[16 + c0]; vsc[1] = sc[16 + c0 + 1]; vsc[2] = sc[24 + c0]; vsc[3] = sc[24 + c0 + 1];
#pragma unroll
          for (int nt = 0; nt < 2; ++nt) {
            const int r = nt * 8 + ra;
#pragma unroll
            for (int q4 = 0; q4 < D / 64; ++q4) {                         // 16 bytes: four steps of the contraction
              const uint4 x = *reinterpret_cast<const uint4*>(k_tile + r * S::kRow + (((tl * (D / 64) + q4) ^ (r & 1)) * 16));
              const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
              for (int i = 0; i < 4; ++i)
                mma16816<T>(s[nt], qf[q4 * 4 + i], widen<T>(__byte_perm(w[i], 0u, 0x4140)), widen<T>(__byte_perm(w[i], 0u, 0x4342)));
            }
          }
        }
        // ---- scale, cap, bias, mask
        float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int e = 0; e < 2 * H; ++e) {
            const int col = tok0 + nt * 8 + 2 * tl + (e & 1), h = e >> 1;
            float v = s[nt][e] * ksc[nt * 2 + (e & 1)];
            if (p.softcap > 0.f) v = softcap_score(v * p.scale, p.softcap) * kLog2e;
            else v *= scale2;
            v += al[h] * (float)(col - (kv_len - 1));
            if (p.bias) {
              const int dist = kv_len - 1 - col;
              v += (dist >= p.bias_len - 1 || bs[h] == nullptr) ? far[h] : bs[h][max(0, dist)] * kLog2e;
            }
            if (!live[h] || col >= kv_len || col < lo_pos) v = -INFINITY;
            s[nt][e] = v;
            mx[h] = fmaxf(mx[h], v);
          }
        float corr[2] = {1.f, 1.f}, ms[2];
#pragma unroll
        for (int h = 0; h < H; ++h) {
          mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 1));
          mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 2));
          const float mn = sigmoid ? 0.f : fmaxf(m[h], mx[h]);
          ms[h] = mn == -INFINITY ? 0.f : mn;
          corr[h] = exp2f(m[h] - ms[h]);                                  // (m = -inf: 0)
          m[h] = mn;
        }
        uint32_t pf[4] = {0u, 0u, 0u, 0u};
#pragma unroll
        for (int h = 0; h < H; ++h) {
          float rs = 0.f, pv[2][2];
#pragma unroll
          for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const float x = s[nt][2 * h + e];
              const float pe = sigmoid ? __fdividef(1.f, 1.f + exp2f(-x - sh[h])) : exp2f(x - ms[h]);
              rs += pe;
              pv[nt][e] = pe * vsc[nt * 2 + e];
            }
          pf[h] = pack2<T>(pv[0][0], pv[0][1]);
          pf[2 + h] = pack2<T>(pv[1][0], pv[1][1]);
          rs += __shfl_xor_sync(0xffffffffu, rs, 1);
          rs += __shfl_xor_sync(0xffffffffu, rs, 2);
          l[h] = l[h] * corr[h] + rs;
        }
        if (__any_sync(0xffffffffu, corr[0] != 1.f || corr[1] != 1.f)) {
#pragma unroll
          for (int i = 0; i < ND; ++i) {
            o[i][0] *= corr[0]; o[i][1] *= corr[0];
            if (H > 1) { o[i][2] *= corr[1]; o[i][3] *= corr[1]; }
          }
        }
        if constexpr (KIND == 0) {
#pragma unroll
          for (int i = 0; i < ND; i += 2) {
            uint32_t vf[4];
            const int mat = lane >> 3, r = (mat & 1) * 8 + (lane & 7);
            ldmatrix_x4_trans(vf, v_tile + r * S::kRow + (((i + (mat >> 1)) ^ (r & 7)) * 16));
            mma16816<T>(o[i], pf, vf[0], vf[1]);
            mma16816<T>(o[i + 1], pf, vf[2], vf[3]);
          }
        } else {
          // lane (g = ra, t = tl): columns 16 g .. of tokens 2t, 2t + 1, 2t + 8, 2t + 9
          uint4 x[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int r = 2 * tl + (j & 1) + (j >> 1) * 8;
            x[j] = *reinterpret_cast<const uint4*>(v_tile + r * S::kRow + ((ra ^ (((r >> 1) & 3) << 1)) * 16));
          }
#pragma unroll
          for (int i = 0; i < ND; ++i) {
            auto word = [&](const uint4& v) { return i / 4 == 0 ? v.x : i / 4 == 1 ? v.y : i / 4 == 2 ? v.z : v.w; };
            const uint32_t sel = (uint32_t)((4 + i % 4) << 8 | (i % 4));
            mma16816<T>(o[i], pf, widen<T>(__byte_perm(word(x[0]), word(x[1]), sel)), widen<T>(__byte_perm(word(x[2]), word(x[3]), sel)));
          }
        }
      }
      __syncwarp();
      stage = (stage + 1) % kStages;
    }
    // ---- the sequence's end, or this CTA's: the next queries have landed when the warps have met
    if (u - seg0 < kStages) cp_async_wait<0>();
    // the warps' states meet in warp 0 and go to the first buffer
#pragma unroll 1
    for (int step = 2; step >= 0; --step) {                               // warps 2, 3 to 0, 1; 1 to 0; 0 to memory
      __syncthreads();
      if (step == 2 ? warp >= 2 : warp == step) put(merge[step == 2 ? warp - 2 : step]);
      __syncthreads();
      if (step == 2 ? warp < 2 : step == 1 && warp == 0) add(merge[step == 2 ? warp : 1]);
    }
    if (seg0 == first && seg_end == behind) {
      write(b, 1, merge[0], 0, merge[0]);
    } else {
      const bool tail = seg0 != first;              // the range starts inside the sequence
      float* mine = slot(grp, tail);
      for (int i = tid; i < kSlot / 4; i += kThreads)
        reinterpret_cast<float4*>(mine)[i] = reinterpret_cast<const float4*>(merge[0])[i];
      if (tail) left0 = b; else left1 = b;
    }
    if (u == behind) u += kEnd;
    ++b;
    qb ^= 1;
  }
  cp_async_wait<0>();
  // the sequences that this CTA left parts of, at most its first and its last: was it the last to arrive?
  __syncthreads();
  const int left = tid == 0 ? left0 : tid == 1 ? left1 : -1;
  if (left >= 0) {
    __threadfence();                                // (the barrier ordered the others' parts before it)
    int c0, c1;
    sharers(left, c0, c1);
    int* at = &counters[left * p.num_kv_heads + hk];
    const bool last = atomicAdd(at, 1) == c1 - c0;
    if (last) *at = 0;                              // (nobody comes after; the next launch finds zero)
    s_done[tid] = last ? left : -1;
  }
  __syncthreads();
#pragma unroll 1
  for (int i = 0; i < 2; ++i) {
    const int seq = s_done[i];
    if (seq < 0) continue;
    __threadfence();
    int c0, c1;
    sharers(seq, c0, c1);
    write(seq, c1 - c0 + 1, slot(c0 + 1, true), (int64_t)p.num_kv_heads * 2 * kSlot, slot(c0, space * c0 / groups > s_pre[seq]));
  }
}

template <typename T, int D, int KIND, int ROWS>
cudaError_t run(const DecodeParams& p, int batch, int sms, float* parts, int* counters, bool early, int64_t* floats, cudaStream_t stream) {
  using S = StreamSmem<D, KIND, ROWS>;
  const int bytes = S::total(batch);
  const int fit = D > 128 ? 1 : KIND == 1 ? 3 : 2, room = 228 * 1024 / (bytes + 1024);
  const int slots = sms * (fit < room ? fit : room), groups = slots / p.num_kv_heads > 1 ? slots / p.num_kv_heads : 1;
  if (floats != nullptr) {
    *floats = (int64_t)groups * p.num_kv_heads * 2 * (S::kState / 4);
    return cudaSuccess;
  }
  auto kern = paged_decode_stream_kernel<T, D, KIND, ROWS>;
  // a per-device attribute of the kernel: set on every launch (cheap) rather than once per process
  const cudaError_t set = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (set != cudaSuccess) return set;
  if (early) return pdl_run(kern, groups * p.num_kv_heads, kThreads, bytes, stream, p, batch, parts, counters);
  kern<<<groups * p.num_kv_heads, kThreads, bytes, stream>>>(p, batch, parts, counters);
  return cudaPeekAtLastError();
}

// Shared memory of the instantiation that `dispatch` takes.
int smem_of(int group, int head, int kind, int batch) {
#define TOTAL(D, K) (group <= 8 ? StreamSmem<D, K, 8>::total(batch) : StreamSmem<D, K, 16>::total(batch))
  if (kind == 1) return TOTAL(128, 1);
  return head <= 64 ? TOTAL(64, 0) : head <= 128 ? TOTAL(128, 0) : TOTAL(256, 0);
#undef TOTAL
}

template <typename T>
cudaError_t dispatch(const DecodeParams& p, int kind, int batch, int sms, float* parts, int* counters, bool early, int64_t* floats,
             cudaStream_t stream) {
  const int g = p.num_q_heads / p.num_kv_heads, head = p.dqk > p.dv ? p.dqk : p.dv;
#define RUN(D, K) (g <= 8 ? run<T, D, K, 8>(p, batch, sms, parts, counters, early, floats, stream) \
                          : run<T, D, K, 16>(p, batch, sms, parts, counters, early, floats, stream))
  if (kind == 1) return RUN(128, 1);
  if (head <= 64) return RUN(64, 0);
  if (head <= 128) return RUN(128, 0);
  return RUN(256, 0);
#undef RUN
}

}  // namespace

// Whether the kernel serves a step of `batch` sequences of one token each.  16 rows of heads wider than 128 would take 240 KB of
// shared memory, of which a CTA may have 227: these stay in attn_decode.cu.  So do most other steps with more than 8 heads per key
// head, which need that kernel's 16 rows anyway: its CTAs, cut into splits for few sequences, fall behind only where they leave an
// uneven last wave, and for int8 rows also when there are many.  us there / here, even rows: 48 heads over 4, 16 rows of 1024 29 /
// 25, 64 rows 39 / 54; int8, 32 heads over 2: 8 rows of 4096 26 / 30, 64 rows 132 / 80, 128 rows of 1024 53 / 56, 256 rows 103 / 86.
bool decode_stream_serves(const DecodeParams& p, int kv_kind, int batch, int sms) {
  const int head = p.dqk > p.dv ? p.dqk : p.dv, ctas = batch * p.num_kv_heads;
  if (p.num_q_heads > 8 * p.num_kv_heads && (ctas < 64 || (kv_kind == 0 ? head <= 64 || ctas >= sms : ctas >= sms && ctas < 2 * sms)))
    return false;
  if (batch <= 0 || batch > kMaxBatch || p.num_q_heads > 16 * p.num_kv_heads || batch * p.num_kv_heads > kDecodeCounters ||
      p.block_size % kTile != 0 || smem_of(p.num_q_heads / p.num_kv_heads, head, kv_kind, batch) > kMaxSmem)
    return false;
  return kv_kind == 0 ? p.dqk % 8 == 0 && p.dv % 8 == 0 && head <= 256 : kv_kind == 1 && p.dqk == 128 && p.dv == 128;
}

// Scratch: *floats of partial states; counters, one per (sequence, key head), which are zero and are left so.  early: nothing but
// kernels came before in the stream (programmatic dependent launch).
void decode_stream_scratch(const DecodeParams& p, int kv_kind, int dtype, int batch, int sms, int64_t* floats) {
  if (dtype == 0) dispatch<__nv_bfloat16>(p, kv_kind, batch, sms, nullptr, nullptr, false, floats, nullptr);
  else dispatch<__half>(p, kv_kind, batch, sms, nullptr, nullptr, false, floats, nullptr);
}

cudaError_t decode_stream(const DecodeParams& p, int kv_kind, int dtype, int batch, int sms, float* parts, int* counters, bool early,
                          cudaStream_t stream) {
  return dtype == 0 ? dispatch<__nv_bfloat16>(p, kv_kind, batch, sms, parts, counters, early, nullptr, stream)
                    : dispatch<__half>(p, kv_kind, batch, sms, parts, counters, early, nullptr, stream);
}

}  // namespace b200
