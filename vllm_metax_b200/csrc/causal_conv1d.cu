// Depthwise causal convolution over ragged token batches with a per-sequence carry (the short convolution in front
// of gated-delta-rule / Mamba style mixers).
//
//   y[t, c] = act( bias[c] + sum_j w[c, j] * x_ext[t - (K-1) + j, c] ),   j = 0 .. K-1
//
// where x_ext is the sequence's tokens preceded by the K-1 inputs kept from its previous step (zeros for a new
// sequence).  Tokens are flat [T, C] with sequences given by query_start_loc; the carry lives in
// state[slot, K-1, C] (oldest first) and is rewritten by a second kernel once the outputs are done, so a decode step
// (one token) and a prefill chunk (thousands) go through the same two launches.
//
// Forward kernel: a thread takes 8 channels (16 bytes) of 4 or, where the tokens fill the GPU that way, 8 tokens; their rows and
// the K-1 before them are read first, all at once; bound by that traffic.  Rows whose channel count, pitch or base does not allow
// 16-byte reads, and fp32, go through the kernel with a channel per thread, and so do steps of few tokens: with kVecWork outputs
// and less there are too few threads of 8 for their reads to be hidden.  us, a channel per thread / 8 channels, both launches:
// 64 tokens, 8192 channels 14.9 / 15.9; 64, 4096 10.6 / 12.2; 200, 1024 11.2 / 12.5; 200, 4096 16.0 / 14.7; 500, 4096 18.9 / 14.3;
// 3949, 8192 182 / 64.
// The channels may be gathered from rows that hold several heads' q, k, v and gates in turn (`map`): the projection of a
// gated-delta-rule layer is read where it is.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "common.cuh"
#include "ops.h"

namespace b200 {
namespace {

// Where channel c of a row is read: as it is, or from `heads` groups of `group` entries that start with dk of q, dk of k and dv
// of v, while channels are all q, then all k, then all v.
struct ChannelMap {
  int heads, dk, dv, group;                        // heads 0: as it is
  __device__ __forceinline__ int operator()(int c) const {
    if (heads == 0) return c;
    const int nk = heads * dk;
    if (c < nk) return c / dk * group + c % dk;
    c -= nk;
    if (c < nk) return c / dk * group + dk + c % dk;
    c -= nk;
    return c / dv * group + 2 * dk + c % dv;
  }
};

// The largest s with qsl[s] <= t.
__device__ __forceinline__ int sequence_of(const int* __restrict__ qsl, int batch, int t) {
  int lo = 0, hi = batch - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (qsl[mid] <= t) lo = mid; else hi = mid - 1;
  }
  return lo;
}

constexpr int kMaxK = 8, kVecWork = 640 * 1024;

template <typename T>
__device__ __forceinline__ float ld(const T* p) { return (float)*p; }
template <typename T>
__device__ __forceinline__ void st(T* p, float v) { *p = (T)v; }

// kTokPerCta: 32 for prompts; a handful for decode steps, whose few tokens must still fill the GPU.
template <typename T, int kTokPerCta>
__global__ void conv1d_fwd_kernel(T* __restrict__ out, const T* __restrict__ x, int64_t x_stride,
                                  const T* __restrict__ w, const T* __restrict__ bias, const T* __restrict__ state,
                                  const int* __restrict__ qsl, const int* __restrict__ state_idx,
                                  const int* __restrict__ has_init, int batch, int tokens, int channels, int K,
                                  int silu, ChannelMap map) {
  // per token of this CTA's chunk: first token of its sequence, and the carry slot to read (-1: zeros)
  __shared__ int s_start[kTokPerCta];
  __shared__ int s_slot[kTokPerCta];
  const int t0 = blockIdx.y * kTokPerCta;
  const int t1 = min(tokens, t0 + kTokPerCta);
  if (threadIdx.x < kTokPerCta) {
    const int t = t0 + threadIdx.x;
    int start = -1, slot = -1;
    if (t < t1 && t < qsl[batch]) {
      const int lo = sequence_of(qsl, batch, t);
      start = qsl[lo];
      const int sl = state_idx ? state_idx[lo] : -1;
      if (sl >= 0 && state != nullptr && (has_init == nullptr || has_init[lo] != 0)) slot = sl;
    }
    s_start[threadIdx.x] = start;               // -1: padding row after the last sequence, nothing is written
    s_slot[threadIdx.x] = slot;
  }
  __syncthreads();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= channels) return;
  float wr[kMaxK];
#pragma unroll
  for (int j = 0; j < kMaxK; ++j) wr[j] = j < K ? ld(w + (int64_t)c * K + j) : 0.f;
  const float b = bias ? ld(bias + c) : 0.f;
  const int xc = map(c);
#pragma unroll 4
  for (int i = 0; i < kTokPerCta; ++i) {
    const int t = t0 + i;
    const int start = s_start[i];
    if (t >= t1 || start < 0) continue;
    const int slot = s_slot[i];
    float acc = b;
#pragma unroll
    for (int j = 0; j < kMaxK; ++j) {
      if (j >= K) break;
      const int src = t - (K - 1) + j;              // token index of this tap
      float v = 0.f;
      if (src >= start) {
        v = ld(x + (int64_t)src * x_stride + xc);
      } else if (slot >= 0) {
        const int back = start - src;               // 1 .. K-1 tokens before the sequence's first new token
        v = ld(state + ((int64_t)slot * (K - 1) + (K - 1 - back)) * channels + c);
      }
      acc += wr[j] * v;
    }
    if (silu) acc = acc / (1.f + __expf(-acc));
    st(out + (int64_t)t * channels + c, acc);
  }
}

template <typename T, int kTok, int K>
__global__ void __launch_bounds__(128)
conv1d_vec_kernel(T* __restrict__ out, const T* __restrict__ x, int64_t x_stride, const T* __restrict__ w,
                  const T* __restrict__ bias, const T* __restrict__ state, const int* __restrict__ qsl,
                  const int* __restrict__ state_idx, const int* __restrict__ has_init, int batch, int tokens, int channels,
                  int silu, ChannelMap map) {
  const int c = (blockIdx.x * 128 + threadIdx.x) * 8;
  if (c >= channels) return;
  const int t0 = blockIdx.y * kTok, t1 = min(min(tokens, t0 + kTok), qsl[batch]);
  if (t0 >= t1) return;
  float wr[K][8], b[8] = {};
#pragma unroll
  for (int e = 0; e < 8; ++e)
#pragma unroll
    for (int j = 0; j < K; ++j) wr[j][e] = ld(w + (int64_t)(c + e) * K + j);
  if (bias) unpack8<T>(*reinterpret_cast<const uint4*>(bias + c), b);
  x += map(c);
  uint4 rows[kTok + K - 1];                        // the K-1 rows before the first token, then the tokens', all on their way at once
#pragma unroll
  for (int i = 0; i < kTok + K - 1; ++i) {
    const int src = t0 - (K - 1) + i;
    rows[i] = src >= 0 && src < t1 ? *reinterpret_cast<const uint4*>(x + (int64_t)src * x_stride) : make_uint4(0u, 0u, 0u, 0u);
  }
  int s = sequence_of(qsl, batch, t0), start = qsl[s], end = qsl[s + 1];
#pragma unroll
  for (int i = 0; i < kTok; ++i) {
    const int t = t0 + i;
    if (t >= t1) break;
    while (t >= end) { ++s; start = end; end = qsl[s + 1]; }        // (t < qsl[batch]: there is such a sequence)
    float acc[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] = b[e];
#pragma unroll
    for (int j = 0; j < K; ++j) {
      uint4 r = rows[i + j];
      const int src = t - (K - 1) + j;
      if (src < start) {                           // before the sequence: its carry, or zeros
        const int sl = state_idx ? state_idx[s] : -1;
        const bool carry = sl >= 0 && state != nullptr && (has_init == nullptr || has_init[s] != 0);
        r = carry ? *reinterpret_cast<const uint4*>(state + ((int64_t)sl * (K - 1) + (K - 1 + src - start)) * channels + c)
                  : make_uint4(0u, 0u, 0u, 0u);
      }
      float f[8];
      unpack8<T>(r, f);
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] += wr[j][e] * f[e];
    }
    if (silu) {
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] = acc[e] / (1.f + __expf(-acc[e]));
    }
    *reinterpret_cast<uint4*>(out + (int64_t)t * channels + c) = pack8<T>(acc);
  }
}

// One thread per (sequence, channel): the last K-1 entries of [carry | new tokens] become the new carry.
template <typename T>
__global__ void conv1d_state_kernel(T* __restrict__ state, const T* __restrict__ x, int64_t x_stride,
                                    const int* __restrict__ qsl, const int* __restrict__ state_idx,
                                    const int* __restrict__ has_init, int channels, int K, ChannelMap map) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const int s = blockIdx.y;
  if (c >= channels) return;
  const int slot = state_idx[s];
  if (slot < 0) return;
  const int start = qsl[s], n = qsl[s + 1] - start;
  if (n <= 0) return;
  const bool carry = has_init == nullptr || has_init[s] != 0;
  const int xc = map(c);
  T* st_base = state + (int64_t)slot * (K - 1) * channels + c;
  float keep[kMaxK];
#pragma unroll
  for (int j = 0; j < kMaxK - 1; ++j) {
    if (j >= K - 1) break;
    const int pos = n - (K - 1) + j;                // position in the new tokens; negative: still in the old carry
    if (pos >= 0) keep[j] = ld(x + (int64_t)(start + pos) * x_stride + xc);
    else keep[j] = carry ? ld(st_base + (int64_t)(K - 1 + pos) * channels) : 0.f;
  }
#pragma unroll
  for (int j = 0; j < kMaxK - 1; ++j) {
    if (j >= K - 1) break;
    st(st_base + (int64_t)j * channels, keep[j]);
  }
}

template <typename T>
void launch(void* out, const void* x, int64_t x_stride, const void* w, const void* bias, void* state, const int* qsl,
            const int* state_idx, const int* has_init, int batch, int tokens, int channels, int K, int silu, ChannelMap map,
            cudaStream_t stream) {
  const int threads = 128;
#define CONV_FWD(TOK)                                                                                              \
  conv1d_fwd_kernel<T, TOK><<<dim3((channels + threads - 1) / threads, (tokens + TOK - 1) / TOK), threads, 0, stream>>>( \
      (T*)out, (const T*)x, x_stride, (const T*)w, (const T*)bias, (const T*)state, qsl, state_idx, has_init, batch, tokens, \
      channels, K, silu, map)
#define CONV_VEC(TOK, TAPS)                                                                                        \
  conv1d_vec_kernel<T, TOK, TAPS><<<dim3((channels / 8 + threads - 1) / threads, (tokens + TOK - 1) / TOK), threads, 0, stream>>>( \
      (T*)out, (const T*)x, x_stride, (const T*)w, (const T*)bias, (const T*)state, qsl, state_idx, has_init, batch, tokens, \
      channels, silu, map)
#define CONV_TOK(TAPS)                                                                                             \
  if ((int64_t)tokens * channels <= (1 << 22)) CONV_VEC(4, TAPS);                                                  \
  else CONV_VEC(8, TAPS)
  bool vec = false;
  if constexpr (sizeof(T) == 2) {
    auto wide = [](const void* at) { return (reinterpret_cast<uintptr_t>(at) & 15) == 0; };
    vec = channels % 8 == 0 && x_stride % 8 == 0 && map.dk % 8 == 0 && map.dv % 8 == 0 && map.group % 8 == 0 && wide(x) &&
          wide(out) && wide(bias) && wide(state) && K >= 2 && K <= 4 && (int64_t)tokens * channels > kVecWork;
    if (vec) {
      if (K == 2) { CONV_TOK(2); }
      else if (K == 3) { CONV_TOK(3); }
      else { CONV_TOK(4); }
    }
  }
  if (!vec) {
    if (tokens <= 64) CONV_FWD(1);
    else if (tokens <= 1024) CONV_FWD(4);
    else CONV_FWD(32);
  }
#undef CONV_FWD
#undef CONV_VEC
#undef CONV_TOK
  if (state != nullptr && state_idx != nullptr && K > 1) {
    dim3 g2((channels + threads - 1) / threads, batch);
    conv1d_state_kernel<T><<<g2, threads, 0, stream>>>((T*)state, (const T*)x, x_stride, qsl, state_idx, has_init,
                                                       channels, K, map);
  }
}

}  // namespace

int causal_conv1d(void* out, const void* x, int64_t x_stride, const void* w, const void* bias, void* state,
                  const int* query_start_loc, const int* state_idx, const int* has_init, int batch, int tokens,
                  int channels, int K, int silu, int heads, int dk, int dv, int group, int dtype, cudaStream_t stream) {
  if (K < 1 || K > kMaxK || batch <= 0 || tokens <= 0) return K < 1 || K > kMaxK ? 1 : 0;
  const ChannelMap map{heads, dk, dv, group};
  if (dtype == 0)
    launch<__nv_bfloat16>(out, x, x_stride, w, bias, state, query_start_loc, state_idx, has_init, batch, tokens,
                          channels, K, silu, map, stream);
  else if (dtype == 1)
    launch<__half>(out, x, x_stride, w, bias, state, query_start_loc, state_idx, has_init, batch, tokens, channels, K,
                   silu, map, stream);
  else
    launch<float>(out, x, x_stride, w, bias, state, query_start_loc, state_idx, has_init, batch, tokens, channels, K,
                  silu, map, stream);
  return 0;
}

}  // namespace b200
