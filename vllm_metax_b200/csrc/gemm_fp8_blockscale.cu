// Block-scaled fp8 (e4m3) GEMM, dense and grouped, on tcgen05 (kind::f8f6f4):
//
//     C[m, n] = sum_kb  a_scale[m, kb] * w_scale[n / 128, kb] * ( A8[m, kb-block] . W8[n, kb-block] )
//
// i.e. DeepSeek-style checkpoints: weights e4m3 with one f32 scale per 128 x 128 block
// (`weight_scale_inv`), activations quantised on the fly 1 x 128 per token.  Because the scales
// change every 128 elements of K, each 128-wide K block is multiplied into a FRESH TMEM buffer
// (4 MMAs of K = 32) and the epilogue warps fold it into fp32 register accumulators with the
// block's scale while the tensor core works on the next blocks (all 512 TMEM columns are buffers).
// Eight epilogue warps: two per quarter of the lanes, each with half of the tile's columns; a buffer is given back as soon as
// it is in registers, the folds go two at a time (f32x2), and the next block's scales are on their way meanwhile.
// Tile 128 x 256, or 128 x 128 where N has few tiles; TMA ring of 128-byte-swizzled [rows x 128 B] tiles.
//
// Dense tiles go down M first within groups of kGroupM row blocks, so that the CTAs of a wave share weights and A stays in L2.
// Where whole tiles leave SMs idle for long the (tile, k block) space is cut into one contiguous range per CTA (stream-K):
// a CTA whose range covers part of a tile leaves an fp32 partial in a slot of its own, and the one that arrives last at the tile
// adds them in CTA order.  Nobody waits.  Where K is cut follows the number of rows: results that must not depend on the batch take
// whole tiles, whose sums run through K in one order whatever the tile.
// Grouped mode: A is the expert-sorted padded activation matrix, W [E, N, K], w_scale
// [E, N/128, K/128]; block_expert / total_padded as in gemm_grouped_tcgen05.cu.  With `sorted_ids`, rows of padding (at a block's
// end) are neither read, folded nor written: with a handful of rows per expert they are most of a block.
// us with 128 threads folding whole tiles of 128 x 128 / now, in a replayed graph: 64 x 2112 x 7168 28.9 / 24.8, 64 x 7168 x 16384
// 61.5 / 41, 2048 x 36864 x 7168 907 / 606; 64 experts 4096 x 7168 for 64 x 8 rows 389 / 300, for 1836 x 8 rows 804 / 680.
// Replaces cutlass_fp8_block_scaled_mm / deep_gemm fp8 grouped GEMMs
// (vllm_metax/model_executor/layers/quantization/_cutlass_ops.py:23-38,
// experts/batched_deep_gemm_moe.py:299-326).
#include "common.cuh"
#include "f32x2.cuh"
#include "ops.h"
#include "ptx_sm100.cuh"
#include "tma_host.h"

namespace b200 {
using namespace ptx;

constexpr int kF8BM = 128, kF8BK = 128, kF8Threads = 320, kF8GroupM = 16, kF8BoxM = 32;

template <int BN>
struct F8Smem {
  static constexpr int kStages = BN == 256 ? 4 : 6;
  static constexpr int kBufs = 512 / BN;
  static constexpr int kABytes = kF8BM * kF8BK;
  static constexpr int kBBytes = BN * kF8BK;
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kBarOffset = kStages * kStageBytes;
  static constexpr int kDyn = kBarOffset + (2 * kStages + 2 * kBufs) * 8 + 32 + 1024;
};

struct F8Params {
  void* C;
  const float *a_scale, *w_scale;
  const int *block_expert, *total_padded, *sorted_ids;
  float* ws;           // stream-K: two slots of 128 x BN floats per CTA
  int* counters;       // one per tile, zero
  int M, N, K, ldc, experts, numel;
  StatusWord* status;
};

enum F8Kind { kF8Dense = 0, kF8Grouped = 1, kF8StreamK = 2 };

// Walks a CTA's share: tiles with their range of k blocks.
template <int KIND>
struct F8Walk {
  int num_tiles, num_k, num_m, num_n;
  long long units, u, u_end;                    // stream-K
  int tile, kb0, kb1;
  __device__ F8Walk(int nm, int nn, int nk) : num_tiles(nm * nn), num_k(nk), num_m(nm), num_n(nn), units(0), u(0), u_end(0) {
    if constexpr (KIND == kF8StreamK) {
      units = (long long)num_tiles * num_k;
      u = units * blockIdx.x / gridDim.x;
      u_end = units * (blockIdx.x + 1) / gridDim.x;
    } else {
      u = blockIdx.x;
    }
  }
  __device__ bool next() {
    if constexpr (KIND == kF8StreamK) {
      if (u >= u_end) return false;
      tile = (int)(u / num_k);
      kb0 = (int)(u % num_k);
      kb1 = (int)min((long long)num_k, kb0 + (u_end - u));
      u += kb1 - kb0;
    } else {
      if (u >= num_tiles) return false;
      tile = (int)u;
      kb0 = 0;
      kb1 = num_k;
      u += gridDim.x;
    }
    return true;
  }
  __device__ void where(int& mb, int& tn) const {
    if constexpr (KIND == kF8Grouped) {
      mb = tile / num_n;
      tn = tile % num_n;
    } else {
      const int per = kF8GroupM * num_n, g = tile / per, first = g * kF8GroupM, in = tile % per;
      const int size = min(kF8GroupM, num_m - first);
      mb = first + in % size;
      tn = in / size;
    }
  }
};

__device__ __forceinline__ void f8_bar_epilogue() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

template <typename T, int BN, int KIND>
__global__ void __launch_bounds__(kF8Threads, 1)
gemm_fp8_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmW, const F8Params p) {
  using L = F8Smem<BN>;
  constexpr bool GROUPED = KIND == kF8Grouped;
  constexpr int kStages = L::kStages, kBufs = L::kBufs, CW = BN / 2;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + L::kBarOffset);
  uint64_t* empty_bar = full_bar + kStages;
  uint64_t* part_full = empty_bar + kStages;
  uint64_t* part_empty = part_full + kBufs;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(part_empty + kBufs);
  volatile int* arrival = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rows = GROUPED ? *p.total_padded : p.M;
  const int sk = ceil_div(p.K, kF8BK);          // k blocks of a tile, scale row length
  const int sn = ceil_div(p.N, 128);
  F8Walk<KIND> walk(ceil_div(rows, kF8BM), ceil_div(p.N, BN), sk);
  constexpr uint32_t kTmemCols = 512;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int i = 0; i < kBufs; ++i) {
      mbar_init(&part_full[i], 1);
      mbar_init(&part_empty[i], 256);
    }
    fence_mbar_init();
    prefetch_tensormap(&tmA);
    prefetch_tensormap(&tmW);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  auto expert_of = [&](int mb) -> int {
    if (!GROUPED) return 0;
    int e = p.block_expert[mb];
    if (e < 0 || e >= p.experts) e = 0;
    return e;
  };
  // 32-row boxes of a row block that hold rows at all (dense: the map ends at M and fills with zeros)
  auto boxes_of = [&](int mb) -> int {
    int n = ceil_div(min(kF8BM, rows - mb * kF8BM), kF8BoxM);
    if (GROUPED && p.sorted_ids != nullptr)
      while (n > 1 && p.sorted_ids[mb * kF8BM + (n - 1) * kF8BoxM] >= p.numel) --n;
    return n;
  };

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      while (ok && walk.next()) {
        int mb, tn;
        walk.where(mb, tn);
        const int e = expert_of(mb), boxes = boxes_of(mb);
        const uint32_t bytes = L::kBBytes + boxes * kF8BoxM * kF8BK;
        for (int kb = walk.kb0; kb < walk.kb1; ++kb) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1)) {
            report_status(p.status, kWaitTimeout, 90, walk.tile, kb);
            ok = false;
            break;
          }
          uint8_t* sa = smem + stage * L::kStageBytes;
          mbar_expect_tx(&full_bar[stage], bytes);
          if (GROUPED) tma_load_3d(sa + L::kABytes, &tmW, &full_bar[stage], kb * kF8BK, tn * BN, e);
          else tma_load_2d(sa + L::kABytes, &tmW, &full_bar[stage], kb * kF8BK, tn * BN);
          for (int i = 0; i < boxes; ++i)
            tma_load_2d(sa + i * kF8BoxM * kF8BK, &tmA, &full_bar[stage], kb * kF8BK, mb * kF8BM + i * kF8BoxM);
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // c = f32, a = b = e4m3 (format code 0)
      constexpr uint32_t idesc = make_idesc(1, 0, 0, kF8BM, BN);
      int stage = 0;
      uint32_t phase = 0;
      uint32_t it = 0;   // running K-block count across tiles selects the partial buffer
      bool ok = true;
      while (ok && walk.next()) {
        for (int kb = walk.kb0; kb < walk.kb1; ++kb, ++it) {
          const int pb = it % kBufs;
          if (!mbar_wait(&part_empty[pb], ((it / kBufs) & 1) ^ 1) || !mbar_wait(&full_bar[stage], phase)) {
            report_status(p.status, kWaitTimeout, 91, walk.tile, kb);
            ok = false;
            break;
          }
          tc_fence_after_sync();
          const uint32_t sa = smem_u32(smem + stage * L::kStageBytes);
          const uint64_t da = make_smem_desc_sw128(sa), db = make_smem_desc_sw128(sa + L::kABytes);
#pragma unroll
          for (int k = 0; k < kF8BK / 32; ++k)
            umma_f8_ss(tmem_base + pb * BN, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc, k != 0 ? 1u : 0u);
          umma_commit(&empty_bar[stage]);
          umma_commit(&part_full[pb]);
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else {
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    uint32_t it = 0;
    bool ok = true;                             // (a warp that gave up still meets the others at their barriers)
    while (walk.next()) {
      int mb, tn;
      walk.where(mb, tn);
      const int e = expert_of(mb);
      const int row = mb * kF8BM + quarter * 32 + lane;
      const bool row_ok = row < rows && !(GROUPED && p.sorted_ids != nullptr && p.sorted_ids[row] >= p.numel);
      const bool busy = __any_sync(0xffffffffu, row_ok);          // (the other quarters only give the buffers back)
      const int col0 = tn * BN + half * CW;
      const float* as = p.a_scale + (size_t)(row_ok ? row : 0) * sk;
      const float* ws = p.w_scale + ((size_t)e * sn + min(col0 / 128, sn - 1)) * sk;
      uint64_t acc[CW / 2];
#pragma unroll
      for (int i = 0; i < CW / 2; ++i) acc[i] = 0ull;
      float sc = busy ? as[walk.kb0] * ws[walk.kb0] : 0.f;
      for (int kb = walk.kb0; ok && kb < walk.kb1; ++kb, ++it) {
        const int pb = it % kBufs;
        float next = 0.f;
        if (busy && kb + 1 < walk.kb1) next = as[kb + 1] * ws[kb + 1];
        if (!mbar_wait(&part_full[pb], (it / kBufs) & 1)) {
          report_status(p.status, kWaitTimeout, 92, walk.tile, kb);
          ok = false;
          break;
        }
        if (busy) {
          tc_fence_after_sync();
          const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + pb * BN + half * CW;
          const uint64_t s2 = pack2f(sc, sc);
#pragma unroll
          for (int c = 0; c < CW; c += 64) {
            uint32_t r[2][32];
            tmem_ld_32x32b_x32(taddr + c, r[0]);
            tmem_ld_32x32b_x32(taddr + c + 32, r[1]);
            tmem_ld_wait();
            if (c + 64 == CW) {
              tc_fence_before_sync();
              mbar_arrive(&part_empty[pb]);
            }
#pragma unroll
            for (int i = 0; i < 64; i += 2)
              acc[(c + i) / 2] = fma2f(pack2f(__uint_as_float(r[i / 32][i % 32]), __uint_as_float(r[i / 32][i % 32 + 1])), s2,
                                       acc[(c + i) / 2]);
          }
        } else {
          mbar_arrive(&part_empty[pb]);
        }
        sc = next;
      }
      if constexpr (KIND == kF8StreamK) {
        if (walk.kb0 != 0 || walk.kb1 != walk.num_k) {
          // slot 0: the tile's first blocks belong to others; a float4 per lane, rows side by side
          const int at = half * (CW / 4) * kF8BM + quarter * 32 + lane;
          if (busy) {
            float4* slot = reinterpret_cast<float4*>(p.ws + ((size_t)blockIdx.x * 2 + (walk.kb0 == 0)) * kF8BM * BN);
#pragma unroll
            for (int i = 0; i < CW / 4; ++i) {
              float4 v;
              unpack2f(acc[2 * i], v.x, v.y);
              unpack2f(acc[2 * i + 1], v.z, v.w);
              slot[at + i * kF8BM] = v;
            }
          }
          __threadfence();
          f8_bar_epilogue();
          const long long first = (long long)walk.tile * walk.num_k, last = first + walk.num_k - 1;
          const int c0 = (int)(((first + 1) * gridDim.x - 1) / walk.units), c1 = (int)(((last + 1) * gridDim.x - 1) / walk.units);
          if (threadIdx.x == 64) *arrival = atomicAdd(&p.counters[walk.tile], 1);
          f8_bar_epilogue();
          const bool mine = *arrival == c1 - c0;
          f8_bar_epilogue();                     // (arrival is rewritten by the next tile)
          if (!mine) continue;
          __threadfence();
          if (busy) {
#pragma unroll
            for (int i = 0; i < CW / 2; ++i) acc[i] = 0ull;
            const uint64_t one = pack2f(1.f, 1.f);
            for (int c = c0; c <= c1; ++c) {
              const bool head = walk.units * c / gridDim.x <= first;
              const float4* slot = reinterpret_cast<const float4*>(p.ws + ((size_t)c * 2 + head) * kF8BM * BN);
#pragma unroll
              for (int i = 0; i < CW / 4; ++i) {
                const float4 v = __ldcg(slot + at + i * kF8BM);
                acc[2 * i] = fma2f(pack2f(v.x, v.y), one, acc[2 * i]);
                acc[2 * i + 1] = fma2f(pack2f(v.z, v.w), one, acc[2 * i + 1]);
              }
            }
          }
        }
      }
      if (ok && row_ok) {
        T* dst = reinterpret_cast<T*>(p.C) + (size_t)row * p.ldc + col0;
#pragma unroll
        for (int v = 0; v < CW / 8; ++v) {
          const int col = col0 + v * 8;
          float f[8];
#pragma unroll
          for (int i = 0; i < 4; ++i) unpack2f(acc[v * 4 + i], f[2 * i], f[2 * i + 1]);
          if (col + 8 <= p.N) {
            *reinterpret_cast<uint4*>(dst + v * 8) = pack8<T>(f);
          } else {
#pragma unroll
            for (int i = 0; i < 8; ++i)
              if (col + i < p.N) dst[v * 8 + i] = from_f<T>(f[i]);
          }
        }
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

template <typename T, int BN, int KIND>
static void launch_f8(const void* A, int lda, const void* W, int E, const F8Params& p, int grid, cudaStream_t stream) {
  CUtensorMap tmA = make_tmap_2d(A, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, p.M, p.K, lda, kF8BoxM, kF8BK);
  CUtensorMap tmW;
  if (KIND == kF8Grouped) {
    uint64_t wd[3] = {(uint64_t)p.K, (uint64_t)p.N, (uint64_t)E};
    uint64_t ws[2] = {(uint64_t)p.K, (uint64_t)p.N * p.K};
    uint32_t wb[3] = {(uint32_t)kF8BK, (uint32_t)BN, 1};
    tmW = make_tmap_nd(W, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, wd, ws, wb, CU_TENSOR_MAP_SWIZZLE_128B);
  } else {
    tmW = make_tmap_2d(W, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, p.N, p.K, p.K, BN, kF8BK);
  }
  auto kern = gemm_fp8_kernel<T, BN, KIND>;
  // a per-device attribute of the kernel: set on every launch (cheap) rather than once per process
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, F8Smem<BN>::kDyn);
  kern<<<grid, kF8Threads, F8Smem<BN>::kDyn, stream>>>(tmA, tmW, p);
}

// Ranges instead of whole tiles cost some 10 us: their counters' memset, the parts' way through memory, the last arriver's sums.
// A k block of a tile takes 0.3 to 0.5 us, so they pay where they make a CTA's longest share at least kF8Saved blocks shorter (with
// at least 4 blocks per CTA; and with two tiles per SM or more, tiles of twice the width are the better way).  us, whole tiles / ranges and the blocks saved: 1 x 7168 x 18432 60 / 41 (90), 64 x 2112 x 7168
// 27.9 / 24.8 (50), 400 x 1536 x 7168 29.1 / 27.5 (38), 129 x 4096 x 7168 28.7 / 29.0 (32), 1000 x 2112 x 7168 32 / 41 (5),
// 64 x 7168 x 2048 12.8 / 20.7 (10).  Returns the CTAs, or 0.
constexpr int kF8Saved = 34;
static int f8_streamk_ctas(int M, int N, int K, int sms) {
  const int64_t tiles = (int64_t)ceil_div(M, kF8BM) * ceil_div(N, 128), num_k = ceil_div(K, kF8BK), units = tiles * num_k;
  const int64_t ctas = units / 4 < sms ? units / 4 : sms;
  const int64_t longest = (tiles + sms - 1) / sms * num_k;
  return ctas > 0 && tiles < 2 * sms && longest * ctas - units >= kF8Saved * ctas ? (int)ctas : 0;
}

void gemm_fp8_scratch(int M, int N, int K, int sms, int64_t* floats, int64_t* counters) {
  const int ctas = f8_streamk_ctas(M, N, K, sms);
  *floats = (int64_t)ctas * 2 * kF8BM * 128;
  *counters = ctas > 0 ? (int64_t)ceil_div(M, kF8BM) * ceil_div(N, 128) : 0;
}

template <typename T>
static void run_f8(const void* A, int lda, const void* W, int E, const F8Params& p, bool grouped, int sms, cudaStream_t stream) {
  if (!grouped && p.ws != nullptr) {
    launch_f8<T, 128, kF8StreamK>(A, lda, W, E, p, f8_streamk_ctas(p.M, p.N, p.K, sms), stream);
    return;
  }
  // 128 x 256 halves what a block reads of A per product, and its tensor-core time is shared-memory bound at 128 x 128: a tile
  // takes 1.55 times as long as one of 128.  It needs enough tiles, and a last wave that does not give that back (two waves or
  // three, 256 x 24576 x 1536: 30 us, 28 us in the narrow tiles; three or five, 1500 x 7168 x 16384: 245 us, 269 us)
  const int64_t tw = (int64_t)ceil_div(p.M, kF8BM) * (p.N / 256), tn = (int64_t)ceil_div(p.M, kF8BM) * ceil_div(p.N, 128);
  const bool wide = p.N % 256 == 0 && tw >= sms && (grouped || ceil_div(tw, sms) * 31 <= ceil_div(tn, sms) * 20);
  const int64_t tiles = (int64_t)ceil_div(p.M, kF8BM) * ceil_div(p.N, wide ? 256 : 128);
  const int grid = tiles < sms ? (int)tiles : sms;
  if (grouped) {
    if (wide) launch_f8<T, 256, kF8Grouped>(A, lda, W, E, p, grid, stream);
    else launch_f8<T, 128, kF8Grouped>(A, lda, W, E, p, grid, stream);
  } else {
    if (wide) launch_f8<T, 256, kF8Dense>(A, lda, W, E, p, grid, stream);
    else launch_f8<T, 128, kF8Dense>(A, lda, W, E, p, grid, stream);
  }
}

// A [M, K] e4m3 (row pitch lda bytes), a_scale [M, K/128]; W [N, K] or [E, N, K] e4m3 contiguous,
// w_scale [(E,) ceil(N/128), K/128].  K must be a multiple of 128.  out_dtype: 0 bf16, 1 fp16.
// sorted_ids: see above, or null.  ws, counters: as gemm_fp8_scratch says (dense), the counters zero; null: whole tiles.
void gemm_fp8_blockscale(const void* A, int M, int lda, const void* W, int E, int N, int K, void* C, int ldc,
                         const float* a_scale, const float* w_scale, const int* block_expert,
                         const int* total_padded, const int* sorted_ids, int numel, float* ws, int* counters, int sms,
                         int grouped, int out_dtype, cudaStream_t stream, void* status) {
  if (M <= 0 || N <= 0) return;
  const F8Params p{C, a_scale, w_scale, block_expert, total_padded, sorted_ids, ws, counters, M, N, K, ldc, E, numel,
                   reinterpret_cast<StatusWord*>(status)};
  if (out_dtype == 0) run_f8<__nv_bfloat16>(A, lda, W, E, p, grouped != 0, sms, stream);
  else run_f8<__half>(A, lda, W, E, p, grouped != 0, sms, stream);
}

}  // namespace b200
