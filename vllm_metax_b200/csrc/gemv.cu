// One to four tokens against a weight: the product as a stream over its rows.
//
//     C[M, N] = A[M, K] . W[N, K]^T (+ bias) (+ residual), or SiLU-gated over interleaved (gate, up) rows;   M <= 4
//
// A CTA owns an equal, contiguous share of the rows; its warps divide K among them, 16 bytes a lane, so that whatever N and K
// are every SM streams the same number of bytes and a row's sum is finished inside one CTA: no partial tiles in memory, no second
// pass, no ring or tensor memory to set up.  Eight rows (four, for three or four tokens) are on their way per warp at a time; the first rows come to L2 while the
// kernel before still runs.  Bound by the weight's bytes with one token; with more the multiply-adds (one per token and entry, on
// the CUDA cores) begin to count, and the tensor-core kernels take over where bindings_core.cpp says.
// M = 1, bf16, N x K, stream-K on CTA pairs / here behind a small kernel of a graph, us: 6144 x 4096 20 / 12, 28672 x 4096 (gated)
// 50 / 39, 4096 x 14336 32 / 24, 4096 x 4096 16.5 / 9.3, 2048 x 2048 12 / 5.5; M = 4: 4096 x 4096 16.6 / 14.3.
#include "common.cuh"
#include "f32x2.cuh"
#include "ops.h"
#include "pdl.cuh"

namespace b200 {
namespace {

constexpr int kMaxWarps = 16;
template <int M> constexpr int rows_of = M <= 2 ? 8 : 4;     // rows on their way per warp

// The two entries of a 16-bit pair as fp32, packed.
template <typename T>
__device__ __forceinline__ uint64_t widen2(uint32_t v);
template <>
__device__ __forceinline__ uint64_t widen2<__nv_bfloat16>(uint32_t v) {
  return pack2f(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
}
template <>
__device__ __forceinline__ uint64_t widen2<__half>(uint32_t v) {
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&v));
  return pack2f(f.x, f.y);
}

template <typename T, int M>
__global__ void __launch_bounds__(kMaxWarps * 32, M == 1 ? 2 : 1)
gemv_kernel(T* C, const T* A, const T* W, const T* bias,
            const T* residual, int N, int K, int lda, int ldw, int ldc, int ldr, int gate) {
  constexpr int kRows = rows_of<M>;
  extern __shared__ float s_part[];                  // [rows of the CTA][M][warps]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int r0 = (int)((int64_t)(N / 2) * blockIdx.x / gridDim.x) * 2;
  const int r1 = blockIdx.x + 1 == gridDim.x ? N : (int)((int64_t)(N / 2) * (blockIdx.x + 1) / gridDim.x) * 2;
  pdl_trigger();
  {
    // the first rows into L2, a line of 128 bytes a thread and step
    const int lines = (K * 2 + 127) / 128;
    for (int i = threadIdx.x; i < lines * kRows; i += blockDim.x) {
      const int r = r0 + i / lines;
      if (r < r1) asm volatile("prefetch.global.L2 [%0];" ::"l"(W + (int64_t)r * ldw + (i % lines) * 64));
    }
  }
  pdl_wait();
  for (int r = r0; r < r1; r += kRows) {
    uint64_t acc[kRows][M];
#pragma unroll
    for (int i = 0; i < kRows; ++i)
#pragma unroll
      for (int m = 0; m < M; ++m) acc[i][m] = 0ull;
    const int n = min(kRows, r1 - r);
    const T* at = W + (int64_t)r * ldw;
#pragma unroll 1
    for (int k = (warp * 32 + lane) * 8; k < K; k += nw * 256) {
      uint4 w[kRows], x[M];
#pragma unroll
      for (int i = 0; i < kRows; ++i) {
        w[i] = make_uint4(0u, 0u, 0u, 0u);
        if (i < n) w[i] = __ldcs(reinterpret_cast<const uint4*>(at + (int64_t)i * ldw + k));
      }
#pragma unroll
      for (int m = 0; m < M; ++m) x[m] = *reinterpret_cast<const uint4*>(A + (int64_t)m * lda + k);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        uint64_t xv[M];
#pragma unroll
        for (int m = 0; m < M; ++m) xv[m] = widen2<T>(e == 0 ? x[m].x : e == 1 ? x[m].y : e == 2 ? x[m].z : x[m].w);
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
          const uint64_t wv = widen2<T>(e == 0 ? w[i].x : e == 1 ? w[i].y : e == 2 ? w[i].z : w[i].w);
#pragma unroll
          for (int m = 0; m < M; ++m) acc[i][m] = fma2f(wv, xv[m], acc[i][m]);
        }
      }
    }
    // the rows' sums per token over the lanes: halve the rows until one is left, then lanes of the same row
#pragma unroll
    for (int m = 0; m < M; ++m) {
      float v[kRows];
#pragma unroll
      for (int i = 0; i < kRows; ++i) {
        float a, b;
        unpack2f(acc[i][m], a, b);
        v[i] = a + b;
      }
      int row = 0, o = 16;
#pragma unroll
      for (int c = kRows / 2; c >= 1; c >>= 1, o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < kRows / 2; ++i)
          if (i < c) v[i] = (up ? v[c + i] : v[i]) + __shfl_xor_sync(0xffffffffu, up ? v[i] : v[c + i], o);
        row += up ? c : 0;
      }
#pragma unroll
      for (; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
      if ((lane & (32 / kRows - 1)) == 0 && row < n) s_part[((r - r0 + row) * M + m) * nw + warp] = v[0];
    }
  }
  __syncthreads();
  auto sum = [&](int row, int m) {
    float v = 0.f;
    for (int w = 0; w < nw; ++w) v += s_part[((row - r0) * M + m) * nw + w];
    return v + (bias ? to_f(bias[row]) : 0.f);
  };
  if (gate) {
    for (int i = threadIdx.x; i < (r1 - r0) / 2 * M; i += blockDim.x) {
      const int row = r0 + i / M * 2, m = i % M;
      const float g = to_f(from_f<T>(sum(row, m))), u = to_f(from_f<T>(sum(row + 1, m)));
      C[(int64_t)m * ldc + row / 2] = from_f<T>(g / (1.f + __expf(-g)) * u);
    }
    return;
  }
  for (int i = threadIdx.x; i < (r1 - r0) * M; i += blockDim.x) {
    const int row = r0 + i / M, m = i % M;
    float v = sum(row, m);
    if (residual) v += to_f(residual[(int64_t)m * ldr + row]);
    C[(int64_t)m * ldc + row] = from_f<T>(v);
  }
}

template <typename T, int M>
void launch(void* C, const void* A, const void* W, const void* bias, const void* residual, int N, int K, int lda, int ldw, int ldc,
            int ldr, int gate, int sms, cudaStream_t stream) {
  int best = 8;                                      // warps: as many as divide K's 256-entry pieces with the least left over
  double idle = 1e9;
  const int pieces = (K + 255) / 256;
  for (int w = kMaxWarps; w >= 8; --w) {
    const int rounds = (pieces + w - 1) / w;
    const double e = (double)rounds * w / pieces - 1 + (kMaxWarps - w) * 0.01;
    if (e < idle - 1e-9) { idle = e; best = w; }
  }
  int grid = sms * (M == 1 ? 2 : 1);
  if (grid > N / 8) grid = N / 8 > 0 ? N / 8 : 1;
  const size_t smem = (size_t)(N / grid + 4) * M * best * sizeof(float);
  auto kern = gemv_kernel<T, M>;
  if (smem > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  pdl_run(kern, grid, best * 32, smem, stream, (T*)C, (const T*)A, (const T*)W, (const T*)bias, (const T*)residual, N, K, lda, ldw,
          ldc, ldr, gate);
}

}  // namespace

// Returns 0, or 1 where another kernel has to do it: more than 4 tokens, rows not on 16 bytes, too many rows for a CTA's sums.
int gemv(void* C, const void* A, const void* W, const void* bias, const void* residual, int M, int N, int K, int lda, int ldw,
         int ldc, int ldr, int gate, int dtype, int sms, cudaStream_t stream) {
  auto wide = [](const void* at) { return (reinterpret_cast<uintptr_t>(at) & 15) == 0; };
  if (M < 1 || M > 4 || K % 8 || lda % 8 || ldw % 8 || !wide(A) || !wide(W) || N < 2 || (gate && (N % 2 || residual)) ||
      (int64_t)(N / sms + 8) * 4 * kMaxWarps * 4 > 100 * 1024)
    return 1;
#define GEMV(T, MM) launch<T, MM>(C, A, W, bias, residual, N, K, lda, ldw, ldc, ldr, gate, sms, stream)
#define GEMV_M(T) if (M == 1) GEMV(T, 1); else if (M == 2) GEMV(T, 2); else if (M == 3) GEMV(T, 3); else GEMV(T, 4)
  if (dtype == 0) { GEMV_M(__nv_bfloat16); } else { GEMV_M(__half); }
#undef GEMV_M
#undef GEMV
  return 0;
}

}  // namespace b200
