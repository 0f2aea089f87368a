// What stands between the projections and the attention of a latent-attention layer (DeepSeek sizes: 512 + 64 entries in the
// cache, 128 + 64 per query head), one launch each:
//
//   mla_rope_insert   per token: RMS norm of the latent, rotation of the shared key part and of every query head's (pairs
//                     (2i, 2i + 1)), the cache row, and for rows that attend in the absorbed form the rotated part behind the
//                     place of the absorbed queries
//   mla_expand_keys   keys of a prompt: a head's own part from the up-projection beside the shared rotated one
//
// Both are bound by their bytes: 16 bytes a thread and access.  What they replace (a norm, a
// rotation, the cache write and copies) took 54 us for 64 decode rows and 590 us for 1836 rows of prompts with 128 heads; they 4 and 55.
#include "common.cuh"
#include "ops.h"

namespace b200 {
namespace {

constexpr int kLat = 512, kRot = 64, kThreads = 256;

// Pairs (2i, 2i + 1) of 8 entries from c on; cs: 32 cosines, then 32 sines.
__device__ __forceinline__ void rotate8(float (&f)[8], const float* __restrict__ cs, int c) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float co = cs[c / 2 + i], si = cs[kRot / 2 + c / 2 + i], a = f[2 * i], b = f[2 * i + 1];
    f[2 * i] = a * co - b * si;
    f[2 * i + 1] = b * co + a * si;
  }
}

template <typename T>
__global__ void __launch_bounds__(kThreads)
mla_rope_insert_kernel(const MlaRopeInsertParams p) {
  __shared__ __align__(16) float s_cs[kRot];
  __shared__ float s_sum[2];
  const int64_t t = blockIdx.x;
  const int tid = threadIdx.x;
  if (tid < kRot / 4)
    reinterpret_cast<float4*>(s_cs)[tid] = reinterpret_cast<const float4*>(p.cos_sin + p.positions[t] * kRot)[tid];
  const T* row = reinterpret_cast<const T*>(p.kv) + t * p.kv_stride;
  float f[8];
  if (tid < kLat / 8 && blockIdx.y == 0) {
    float ss = 0.f;
    unpack8<T>(*reinterpret_cast<const uint4*>(row + tid * 8), f);
#pragma unroll
    for (int i = 0; i < 8; ++i) ss += f[i] * f[i];
    ss = warp_sum(ss);
    if ((tid & 31) == 0) s_sum[tid >> 5] = ss;
  }
  __syncthreads();
  if (blockIdx.y == 0 && tid < (kLat + kRot) / 8) {
    int64_t slot = p.slots[t];
    if (slot >= p.num_slots) {
      if (tid == 0) report_status(p.status, kBadIndex, 11, (int)p.num_slots, (int)slot);
      slot = -1;
    }
    if (tid < kLat / 8) {
      const float inv = rsqrtf((s_sum[0] + s_sum[1]) / (float)kLat + p.eps);
      float w[8];
      unpack8<T>(*reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(p.norm_w) + tid * 8), w);
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] = f[i] * inv * w[i];
    } else {
      unpack8<T>(*reinterpret_cast<const uint4*>(row + tid * 8), f);
      rotate8(f, s_cs, tid * 8 - kLat);
    }
    const uint4 v = pack8<T>(f);
    if (slot >= 0) *reinterpret_cast<uint4*>(reinterpret_cast<T*>(p.cache) + slot * (kLat + kRot) + tid * 8) = v;
    if (tid < kLat / 8) *reinterpret_cast<uint4*>(reinterpret_cast<T*>(p.kv_c) + t * kLat + tid * 8) = v;
    else *reinterpret_cast<uint4*>(reinterpret_cast<T*>(p.k_pe) + t * kRot + tid * 8 - kLat) = v;
  }
  // query heads: 8 lanes each
  const int per = (p.heads + gridDim.y - 1) / gridDim.y, h1 = min(p.heads, ((int)blockIdx.y + 1) * per);
  for (int h = blockIdx.y * per + tid / 8; h < h1; h += kThreads / 8) {
    const int c = tid % 8 * 8;
    T* q = reinterpret_cast<T*>(p.q) + (t * p.heads + h) * p.q_dim + p.q_dim - kRot + c;
    float g[8];
    unpack8<T>(*reinterpret_cast<const uint4*>(q), g);
    rotate8(g, s_cs, c);
    const uint4 v = pack8<T>(g);
    *reinterpret_cast<uint4*>(q) = v;
    if (t < p.absorbed) *reinterpret_cast<uint4*>(reinterpret_cast<T*>(p.qa) + (t * p.heads + h) * (kLat + kRot) + kLat + c) = v;
  }
}

// out [T, heads, nope + 64] = (kv [T, heads, kv_dim] up to nope | k_pe [T, 64]): a thread per 16 bytes of out
__global__ void __launch_bounds__(kThreads)
mla_expand_keys_kernel(uint4* __restrict__ out, const uint4* __restrict__ kv, const uint4* __restrict__ k_pe, int64_t n, int heads,
                       int nope8, int kv8) {
  const int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (i >= n) return;
  const int row8 = nope8 + kRot / 8;
  const int64_t th = i / row8;
  const int c = (int)(i % row8);
  out[i] = c < nope8 ? kv[th * kv8 + c] : k_pe[(th / heads) * (kRot / 8) + c - nope8];
}

}  // namespace

void mla_rope_insert(const MlaRopeInsertParams& p, int dtype, cudaStream_t stream) {
  if (p.tokens <= 0) return;
  const dim3 grid((unsigned)p.tokens, p.tokens >= 512 ? 1 : 4);   // (few tokens: a token's heads over four CTAs)
  if (dtype == 0) mla_rope_insert_kernel<__nv_bfloat16><<<grid, kThreads, 0, stream>>>(p);
  else mla_rope_insert_kernel<__half><<<grid, kThreads, 0, stream>>>(p);
}

void mla_expand_keys(void* out, const void* kv, const void* k_pe, int64_t tokens, int heads, int nope, int kv_dim,
                     cudaStream_t stream) {
  const int64_t n = tokens * heads * ((nope + kRot) / 8);
  if (n <= 0) return;
  mla_expand_keys_kernel<<<(unsigned)((n + kThreads - 1) / kThreads), kThreads, 0, stream>>>(
      (uint4*)out, (const uint4*)kv, (const uint4*)k_pe, n, heads, nope / 8, kv_dim / 8);
}

}  // namespace b200
